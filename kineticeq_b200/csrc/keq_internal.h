// keq_internal.h -- host-side helpers shared by the library's .cu files.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "../../include/keq_b200.h"

// Remember the last CUDA error of the calling thread for keq_last_cuda_error().
void keq_internal_set_cuda_error(cudaError_t e);

// Rows of a row block of the implicit rows kernel at most.
#define KEQ_ROWS_MAX 32

// Host object behind the opaque keq_plan of the C ABI, shared by the
// persistent step kernels (implicit and HOLO).  A plan launches one or more
// kernels per step (`part`), each over a contiguous run of the instance
// records; a part's device header `dev` starts with a keq::PlanHead, and
// `clear_bytes` from `clear` on (the header's barrier and error word last) are
// zeroed before every launch.  Records are `inst_bytes` each, stored in the
// order of the parts (`perm` maps the caller's index to the record), and hold
// their f_in / f_out pointers at the given byte offsets.
enum { KEQ_PLAN_IMPLICIT = 0, KEQ_PLAN_HOLO = 1 };
struct keq_plan_part {
    void* dev;
    void* clear;
    size_t clear_bytes;
    const void* kernel;
    size_t smem;
    int threads;
    int grid;
};
struct keq_plan {
    int kind;
    std::vector<keq_plan_part> part;
    void* dev_inst;
    std::vector<unsigned char> host_inst;
    std::vector<int> perm;
    size_t inst_bytes;
    size_t off_f_in, off_f_out;
    int n_inst;
    int device;
};

// Sets part->grid to every resident CTA of part->kernel (occupancy query).
// smem_limit is the largest dynamic shared memory that any plan launches this
// kernel with: the limit is the kernel's, not the plan's.
keq_status keq_internal_part_grid(keq_plan_part* part, size_t smem_limit);

namespace keq {
// Row-block kernels of the implicit step (keq_implicit_rows.cu,
// keq_implicit_solo.cu) and their dynamic shared memory for a number of warps,
// partial-sum slots and instances / with or without an Anderson ring; 16-byte
// units of the solo kernel's block records.
const void* implicit_rows_entry(int threads, bool aa);
size_t implicit_rows_smem(int warps, int nslot, int n_inst, int buf_rows);
const void* implicit_solo_entry(int conv_type, int aa_on, bool ahead);
size_t implicit_solo_smem(int warps, int nslot, int ring);
size_t implicit_solo_gather_units(int nblk);
// The same of the HOLO step (keq_holo_rows.cu).
const void* holo_rows_entry();
size_t holo_rows_smem(int warps, int nslot, int lo_n);
size_t holo_rows_lorec_units(int lo_n);

// Batched tridiagonal solve (keq_gtsv.cu); scratch: n * batch doubles that a
// call overwrites before reading.
cudaError_t launch_gtsv(const double* dl, const double* d, const double* du, double* B, int n,
                        int batch, double* scratch, cudaStream_t s);
}  // namespace keq
