// keq_implicit_rows.cu -- the implicit (Picard + Anderson) step with one CTA
// per row block: ONE persistent cooperative kernel per time step.
//
// Same method and results as keq_implicit.cu (see there for the reference
// lines); the work is cut differently.  An item is one block of up to 32
// consecutive interior rows of one instance with ALL its velocities; a CTA
// carries an item through a whole Picard iteration, a warp taking tiles of 32
// velocities (one per lane) by the block's rows:
//   1. Maxwellian, assembly and the recurrence with zero inflow, composing
//      the block's map x_out = P x_in + Y per velocity; (P, Y) is published;
//   2. the inflow X is folded from the neighbouring blocks' maps, nearest
//      first: X = Y_1 + P_1 (Y_2 + P_2 (...)), until what is left out cannot
//      change X (see fold_carry).  Maps do not depend on any other block, so
//      there is no chain along x: every block publishes at once and a fold
//      ends after the few blocks that the decay of P leaves visible;
//   3. rows are corrected by P X where that is visible, written, compared
//      with the previous iterate, and summed over the velocities.
// The row moments are complete inside the CTA, which updates W, the Anderson
// history and the next coefficients itself.  One grid barrier ends the
// iteration (convergence is a maximum over all blocks).
//
// This kernel runs plans of several instances and instances with more blocks
// than are resident; keq_implicit_solo.cu runs one resident instance.
//
// What bounds it: the fixed cost of a tile.  In a batch of 64 instances (8-row
// blocks mostly) a tile of 8 rows takes 1130 SM-cycles and one of 32 rows 2660,
// where the FP64 pipe would allow 22 a row; the SMs issue on 36% of the cycles,
// and a warp waits 4.3 cycles per instruction for its CTA (row update), 3.1 for
// memory and 2.3 for dependent arithmetic.  us per step of the batch: 2800 with
// the look-back kernel, 1790 now.  An 8-row block pays for its record, coefficients,
// row update and, with Anderson, history as often as a block of 32 rows (cycles an
// item with Anderson: record 4700, coefficients 10400, sweep 17000, update 4700, Gram
// partials 2800), so batches of small instances want tall blocks (tile_rows), and
// those of at most two velocity tiles run in CTAs of two warps.  us per step of 64
// instances of 200 to 700 rows and 20 to 33 velocities: look-back 441, four warps 614,
// two warps 509, two warps and 24 rows 321; with Anderson 926, 2250, 1570, 826.  Of
// 700 to 2000 rows and 100 to 500 velocities (four warps): look-back 6195, rows by the
// rule 4282, 24 rows 2899; with Anderson 13372, 11130, 6730.
//
// Bounds.  x_i is a convex combination of f^n_i, M_i and x_{i-1} (weights
// 1/d, (dt/tau)/d, cpl/d with d = 1 + dt/tau + cpl), so no |x| exceeds
// G = max(max |f^n|, max M), and a_i = cpl/d <= cpl/(1 + cpl) < 1.  Plan
// creation admits an instance to this kernel when a product of a_max over at
// most kRowsKmax blocks is below 2^-200 (rows_eligible); beyond that the
// look-back kernel runs.
#include <cuda_runtime.h>

#include "keq_rows.cuh"

namespace keq {
namespace rows {

// Tile buffers of a CTA; finish_item and its helpers use them as 32 rows.
__host__ __device__ constexpr size_t bufs_bytes(int warps, int rows) {
    return warps * buf_bytes(rows) > buf_bytes(kRows) ? warps * buf_bytes(rows) : buf_bytes(kRows);
}

constexpr int kListMax = 512;  // instances of a plan that the active list holds

struct alignas(16) CtaSmem : BlockSmem {
    double red[kSlots][2];
    double gbound, nm;
    double gs[kMaxPairs];  // Gram matrix
    unsigned next[2];  // claimed list position, by parity of the claim
    int n_act, act_items;  // active instances of the iteration and their items
    int bad;
    int ok;  // outcome of the grid barrier
};

// The same for the rows of a block and for another CTA (HBM).
__device__ __forceinline__ void save_coef(CtaSmem& C, int i, int k, int nr, const double* c4) {
    const ImpInst& I = C.I;
    reinterpret_cast<double2*>(&I.Wc[4 * (size_t)i])[0] = make_double2(c4[0], c4[1]);
    reinterpret_cast<double2*>(&I.Wc[4 * (size_t)i])[1] = make_double2(c4[2], c4[3]);
    put_coef(C, k, nr, c4);
}

// Row coefficients of W^(m) for the item's rows (warp 0, lane = row) into
// C.coef, and the bound of the fold.  After an applied Anderson call the
// combination is formed here from the history in HBM.
template <bool kAA>
__device__ __noinline__ void stage_rows_coef(CtaSmem& C, int blk, int m, bool cached) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int nx = I.nx, n_inner = I.n_inner;
    const int k0 = blk * I.rblk;
    const int nr = n_inner - k0 < I.rblk ? n_inner - k0 : I.rblk;
    const bool comb = kAA && m >= 1 && aa_applies(I, m - 1);
    const double fmx = ld_cg(&I.scal[0]);
    const double cm = ld_cg(&I.scal[1]), nm = ld_cg(&I.scal[2 + m]);
    const uint2 span = __ldcg(reinterpret_cast<const uint2*>(&I.nanspan[2 * m]));
    double asum = 1.0;
    if (comb) {
        const int d = 3 * n_inner;
        const int mh = m < I.aa_cols ? m : I.aa_cols;
        const int head_out = m % I.aa_cols;
        const int kc = lane < nr ? k0 + lane : k0, i = kc + 1;
        // every load is issued unconditionally (entries past the history length
        // repeat its last column and are selected out of the sums)
        double al[kMaxAACols];
        int col[kMaxAACols];
        const int col0 = ((head_out - mh) % I.aa_cols + I.aa_cols) % I.aa_cols;
#pragma unroll
        for (int jj = 0; jj < kMaxAACols; ++jj) {
            const int jc = jj < mh ? jj : mh - 1;
            al[jj] = ld_cg(&I.alpha[(size_t)(m - 1) * kMaxAACols + jc]);
            col[jj] = col0 + jc >= I.aa_cols ? col0 + jc - I.aa_cols : col0 + jc;
        }
        double acc[3], wnew[3], gv[3][kMaxAACols];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            wnew[q] = ld_cg(&I.Wn[q * nx + i]);
#pragma unroll
            for (int jj = 0; jj < kMaxAACols; ++jj)
                gv[q][jj] = ld_cg(&I.aaG[(size_t)col[jj] * d + q * n_inner + kc]);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            acc[q] = 0.0;
#pragma unroll
            for (int jj = 0; jj < kMaxAACols; ++jj) acc[q] = fma(jj < mh ? gv[q][jj] : 0.0, al[jj], acc[q]);
        }
#pragma unroll
        for (int jj = 0; jj < kMaxAACols; ++jj) asum += jj < mh ? fabs(al[jj]) : 0.0;
        double w3[3], c4[4];
        combine_row(I, acc, wnew, w3, c4);
        if (lane < nr) {
            I.W[i] = w3[0];
            I.W[nx + i] = w3[1];
            I.W[2 * nx + i] = w3[2];
            put_coef(C, lane, nr, c4);
        }
    } else if (!cached && lane < nr) {
        const size_t i = (size_t)(k0 + lane + 1);
        const double2 c01 = __ldcg(reinterpret_cast<const double2*>(&I.Wc[4 * i]));
        const double2 c23 = __ldcg(reinterpret_cast<const double2*>(&I.Wc[4 * i + 2]));
        const double c4[4] = {c01.x, c01.y, c23.x, c23.y};
        put_coef(C, lane, nr, c4);
    }
    if (lane == 0) {
        C.gbound = fold_bound(fmx, cm, nm, m, asum);
        C.nm = nm;
    }
    if ((span.x | span.y) != 0u) {
        __syncwarp();
        if (lane == 0 && I.nblk - (int)span.y < blk) nan_inflow(C, 0);
        if (lane == 1 && (int)span.x - 1 > blk) nan_inflow(C, 1);
    }
}

// Block blk has NaN rows in W^(m) (one thread).
__device__ __forceinline__ void mark_nan(const ImpInst& I, int m, int blk) {
    atomicMax(&I.nanspan[2 * m], (unsigned)(blk + 1));
    atomicMax(&I.nanspan[2 * m + 1], (unsigned)(I.nblk - blk));
}

// Residual maxima and the non-finite flag of an item (warp 1).
__device__ __forceinline__ void flush_residuals(CtaSmem& C, int m) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (I.conv_type == 0) {
        const double r1 = warp_max_bits(lane < nw ? C.red[lane][0] : 0.0);
        const double r2 = warp_max_bits(lane < nw ? C.red[lane][1] : 0.0);
        if (lane == 0) {
            atomic_max_nonneg(&I.res[2 * m], r1);
            atomic_max_nonneg(&I.res[2 * m + 1], r2);
        }
    }
    if (lane == 0 && C.bad) {
        atomicOr(&I.nonfin[m], 1);
        C.bad = 0;
    }
}

// End of an item's sweep (warp 0, lane = row): moments of the new iterate, "w"
// residual, Anderson history, W and coefficients of the next iteration
// (keq_implicit.cu reduce_block has the reference lines).  nm: largest n of the
// iterates before.  In an applied Anderson call the newest residual column goes to
// w.a[row][3 j + q] (the older ones: older_columns).
template <bool kAA>
__device__ __noinline__ void finish_item(CtaSmem& C, TileBuf& w, const double (*part)[3][32], int blk,
                                         int m, double nm, int smask) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int k0 = blk * I.rblk, k = k0 + lane;
    const int nr = I.n_inner - k0 < I.rblk ? I.n_inner - k0 : I.rblk;
    const bool ok = lane < nr;
    const int i = k + 1;
    const int nx = I.nx, n_inner = I.n_inner, d = 3 * n_inner;
    const int nt = I.nvt <= smask ? I.nvt : smask + 1;
    const double s0 = slot_sum<3>(part, nt, 0), s1 = slot_sum<3>(part, nt, 1), s2 = slot_sum<3>(part, nt, 2);
    if (m + 1 < I.picard_iter) {  // largest n of the iterates so far (rounded up to its high word)
        const double mx = n_bound(ok, s0 * I.dv);
        if (lane == 0) atomic_max_nonneg(&I.scal[2 + m + 1], mx > nm ? mx : nm);
    }
    if (any_nan_row(ok, s0 * I.dv) && lane == 0) mark_nan(I, m + 1, blk);
    const bool aa_now = kAA && aa_applies(I, m);
    const bool need_old = I.conv_type == 1 || (kAA && I.aa_on);
    double wn[3] = {0.0, 0.0, 0.0}, wo[3] = {0.0, 0.0, 0.0}, c4[4];
    if (ok) {
        if (need_old) {
            wo[0] = ld_cg(&I.W[i]);
            wo[1] = ld_cg(&I.W[nx + i]);
            wo[2] = ld_cg(&I.W[2 * nx + i]);
        }
        moments_and_coeffs(s0, s1, s2, I.dv, I.dt, I.tau_tilde, 1e-12, wn, c4);
    }
    if (kAA && I.aa_on) {
        const int cols = I.aa_cols;
        const int head_in = m % cols;
        const int mh = (m + 1) < cols ? (m + 1) : cols;
        if (aa_now) {
#pragma unroll
            for (int q = 0; q < 3; ++q) w.a[lane][3 * (mh - 1) + q] = ok ? wn[q] - wo[q] : 0.0;
        }
        if (ok) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                I.Wn[q * nx + i] = wn[q];
                I.aaG[(size_t)head_in * d + q * n_inner + k] = wn[q];
                I.aaR[(size_t)head_in * d + q * n_inner + k] = wn[q] - wo[q];
            }
        }
    }
    if (I.conv_type == 1) {
        FracMax q1, q2;
        if (ok) residual_w(wn, wo, I.abs_tol, I.tol, q1, q2);
        if (blk == 0 && lane < 2) {  // the two boundary rows
            const int ib = lane == 0 ? 0 : nx - 1;
            double b[3], o[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                b[q] = ld_cg(&I.Wb[3 * lane + q]);
                o[q] = ld_cg(&I.W[q * nx + ib]);
            }
            residual_w(b, o, I.abs_tol, I.tol, q1, q2);
        }
        const double r1 = warp_max(frac_value(q1)), r2 = warp_max(frac_value(q2));
        if (lane == 0) {
            atomic_max_nonneg(&I.res[2 * m], r1);
            atomic_max_nonneg(&I.res[2 * m + 1], r2);
        }
    }
    if (!aa_now && ok) {  // bgk1d_implicit_cuda_kernel.py:285-287
        I.W[i] = clamp_min_t(wn[0], 1e-12);
        I.W[nx + i] = wn[1];
        I.W[2 * nx + i] = clamp_min_t(wn[2], 1e-12);
        save_coef(C, i, lane, nr, c4);
    }
    if (blk == 0 && lane < 2) {  // W of the boundary rows: floored moments of the fixed rows
        const int ib = lane == 0 ? 0 : nx - 1;
        I.W[ib] = clamp_min_t(ld_cg(&I.Wb[3 * lane + 0]), 1e-12);
        I.W[nx + ib] = ld_cg(&I.Wb[3 * lane + 1]);
        I.W[2 * nx + ib] = clamp_min_t(ld_cg(&I.Wb[3 * lane + 2]), 1e-12);
    }
    __syncwarp();
}

// The older residual columns of an applied Anderson call into w.a[row][3 j + q], by
// two warps beside finish_item (behind it, one column after another, they cost a
// memory round trip each).  With this, two pairs a warp below, four in
// last_block_alpha and the count of finished blocks beside the next item, 64
// instances of 200 to 700 rows and 20 to 33 velocities, m = 5, took 2250 us a step
// instead of 2480.
__device__ __noinline__ void older_columns(const CtaSmem& C, TileBuf& w, int blk, int m, int half) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int k = blk * I.rblk + lane, n_inner = I.n_inner, d = 3 * n_inner, cols = I.aa_cols;
    const bool ok = lane < I.rblk && k < n_inner;
    const int kc = ok ? k : blk * I.rblk;
    const int head_in = m % cols, mh = (m + 1) < cols ? (m + 1) : cols;
    const int col0 = head_in + 1 >= mh ? head_in + 1 - mh : head_in + 1 - mh + cols;
    double v[kMaxAACols / 2][3];
#pragma unroll
    for (int t = 0; t < kMaxAACols / 2; ++t) {  // clamped: every load is issued
        const int jj = 2 * t + half < mh ? 2 * t + half : 0;
        const int col = col0 + jj >= cols ? col0 + jj - cols : col0 + jj;
#pragma unroll
        for (int q = 0; q < 3; ++q) v[t][q] = ld_cg(&I.aaR[(size_t)col * d + q * n_inner + kc]);
    }
#pragma unroll
    for (int t = 0; t < kMaxAACols / 2; ++t)
        if (2 * t + half < mh - 1)
#pragma unroll
            for (int q = 0; q < 3; ++q) w.a[lane][3 * (2 * t + half) + q] = ok ? v[t][q] : 0.0;
}

// Gram partials of an applied Anderson call over the block's rows: two pairs of
// columns per warp at a time, a lane per row.  After a CTA barrier behind
// finish_item and older_columns.
__device__ __noinline__ void gram_partials(const CtaSmem& C, const TileBuf& w, int blk, int m) {
    const ImpInst& I = C.I;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int mh = (m + 1) < I.aa_cols ? (m + 1) : I.aa_cols;
    const int npairs = mh * (mh + 1) / 2;
    for (int t = warp; t < npairs; t += 2 * nw) {
        const int t2 = t + nw < npairs ? t + nw : t;
        int p, q, p2, q2;
        aa_pair_of(t, mh, p, q);
        aa_pair_of(t2, mh, p2, q2);
        double v = 0.0, v2 = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v = fma(w.a[lane][3 * p + c], w.a[lane][3 * q + c], v);
            v2 = fma(w.a[lane][3 * p2 + c], w.a[lane][3 * q2 + c], v2);
        }
        v = warp_sum(v);
        v2 = warp_sum(v2);
        if (lane == 0) {
            I.gpart[(size_t)t * I.nblk + blk] = v;
            I.gpart[(size_t)t2 * I.nblk + blk] = v2;
        }
    }
}

// Last block of an instance's Anderson call (one warp of its CTA): Gram matrix,
// coefficients into I.alpha.
__device__ __noinline__ void last_block_alpha(CtaSmem& C, int m) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int mh = (m + 1) < I.aa_cols ? (m + 1) : I.aa_cols;
    const int npairs = mh * (mh + 1) / 2;
    for (int t = 0; t < npairs; t += 4) {
        const double* g[4];
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) g[u] = I.gpart + (size_t)(t + u < npairs ? t + u : npairs - 1) * I.nblk;
        aa_pair_sums(g, I.nblk, v);
        if (lane == 0)
#pragma unroll
            for (int u = 0; u < 4; ++u) C.gs[t + u < npairs ? t + u : npairs - 1] = v[u];
    }
    __syncwarp();
    const double al = aa_solve_warp(C.gs, mh, I.aa_reg, I.aa_alpha_max);
    if (lane < mh) I.alpha[(size_t)m * kMaxAACols + lane] = al;
    __syncwarp();
}

// Item of the prologue: moments of f^n, W^(0) and its coefficients, the bounds
// of the fold, empty map slots of both parities.
__device__ __noinline__ void first_item(CtaSmem& C, TileBuf& w, double (*part)[3][32], int blk,
                                        const double* __restrict__ fn, double* __restrict__ fo, int smask) {
    const ImpInst& I = C.I;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int vt = warp; vt < I.nvt; vt += nw) {
        BarrierMaps::clear(BarrierMaps::slot(I, 0, blk, vt));
        BarrierMaps::clear(BarrierMaps::slot(I, 1, blk, vt));
    }
    double mx = warp_max_bits(first_tiles(C, w, part, blk, fn, fo, smask));
    if (lane == 0) C.red[warp][0] = mx;
    __syncthreads();
    if (warp == 0) {
        mx = warp_max_bits(lane < nw ? C.red[lane][0] : 0.0);
        const int nr = I.n_inner - blk * I.rblk < I.rblk ? I.n_inner - blk * I.rblk : I.rblk;
        double n = 0.0, cm = 0.0;
        const int nt = I.nvt <= smask ? I.nvt : smask + 1;
        const double s0 = slot_sum<3>(part, nt, 0);
        if (lane < nr) {
            double w3[3], c4[4];
            moments_and_coeffs(s0, slot_sum<3>(part, nt, 1), slot_sum<3>(part, nt, 2), I.dv, I.dt, I.tau_tilde, 0.0, w3, c4);
            const int i = blk * I.rblk + lane + 1;
            n = w3[0];
            I.W[i] = w3[0];
            I.W[I.nx + i] = w3[1];
            I.W[2 * I.nx + i] = w3[2];
            save_coef(C, i, lane, nr, c4);
            cm = c4[2];
        }
        if (any_nan_row(lane < nr, s0 * I.dv) && lane == 0) mark_nan(I, 0, blk);
        n = warp_max_bits(n);
        cm = warp_max_bits(cm);
        if (lane == 0) {
            atomic_max_nonneg(&I.scal[0], mx);
            atomic_max_nonneg(&I.scal[1], cm);
            atomic_max_nonneg(&I.scal[2], n);
        }
    }
}

// Stage instance b (all threads).
__device__ __forceinline__ void stage_inst(CtaSmem& C, const PlanDev& P, int b, int& cur_b) {
    if (b == cur_b) return;
    __syncthreads();
    const int* s = reinterpret_cast<const int*>(&P.inst[b]);
    int* d = reinterpret_cast<int*>(&C.I);
    for (int q = threadIdx.x; q < (int)(sizeof(ImpInst) / sizeof(int)); q += blockDim.x)
        d[q] = __ldg(s + q);
    cur_b = b;
    __syncthreads();
}

// Items of the instances that are active in iteration m, as a list of runs:
// positions [aoff[q], aoff[q+1]) are the blocks of instance aidx[q].  Every CTA
// builds the same list, so that tickets are spent on active items only (an
// iteration of a batch runs for its slowest instances).  Returns the list's
// length.  All threads; flags by the CTA, the scan by warp 0.
__device__ __forceinline__ int active_list(CtaSmem& C, const PlanDev& P, int n, int m, int* aoff,
                                           unsigned short* aidx) {
    const int lane = threadIdx.x & 31;
    for (int b = threadIdx.x; b < n; b += blockDim.x) aidx[b] = inst_active_rows(P.inst[b], m);
    __syncthreads();
    if (threadIdx.x < 32) {
        int na = 0, tot = 0;
        for (int base = 0; base < n; base += 32) {
            const int b = base + lane;
            const bool on = b < n && aidx[b] != 0;
            const int nb = on ? (int)(__ldg(&P.item_off[b + 1]) - __ldg(&P.item_off[b])) : 0;
            int inc = nb;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                inc += lane >= o ? v : 0;
            }
            const unsigned mk = __ballot_sync(0xffffffffu, on);
            const int pos = na + __popc(mk & ((1u << lane) - 1u));
            __syncwarp();
            if (on) {
                aidx[pos] = (unsigned short)b;  // pos <= b, and b's own flag is consumed
                aoff[pos] = tot + inc - nb;
            }
            na += __popc(mk);
            tot += __shfl_sync(0xffffffffu, inc, 31);
            __syncwarp();
        }
        if (lane == 0) {
            aoff[na] = tot;
            C.n_act = na;
            C.act_items = tot;
        }
    }
    __syncthreads();
    return C.act_items;
}

// kAA: some instance of the plan has Anderson on.  A kernel for each, as the code of
// the calls takes registers from the sweep: batch of 64 without Anderson 1910 -> 1790
// us a step.
template <int kThreads, int kCtas, bool kAA>
__global__ void __launch_bounds__(kThreads, kCtas)
implicit_rows_kernel(PlanDev* __restrict__ Pp, int swap_io) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kClaim = kThreads > 64 ? 64 : 32;  // claims items: not in warp 0
    PlanDev& P = *Pp;
    CtaSmem& C = *reinterpret_cast<CtaSmem*>(smem_raw);
    // the header's constants, read once: every global read behind a barrier is
    // an L2 round trip
    const unsigned G = gridDim.x;
    const int n_inst = P.n_inst, max_iter = P.max_iter, nslot = P.nslot;
    const long long total_items = P.total_items;
    const unsigned long long limit = P.head.spin_limit;
    const bool traced = P.head.trace != nullptr;
    GridBarrier* const bar = &P.head.bar;
    unsigned* const tickets = P.tickets;
    double(*part)[3][32] = reinterpret_cast<double(*)[3][32]>(smem_raw + sizeof(CtaSmem));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    unsigned char* const bufs = reinterpret_cast<unsigned char*>(part + nslot);
    const size_t bstride = buf_bytes(P.buf_rows);
    TileBuf& wbuf = *reinterpret_cast<TileBuf*>(bufs + warp * bstride);
    TileBuf& buf0 = *reinterpret_cast<TileBuf*>(bufs);  // scratch behind the sweeps
    // Four slots do with four warps and up to 16 tiles: the running sum of warp
    // w's tiles w, w+4, ... is the running sum number w of slot_sum.
    const int smask = nw == 4 && nslot <= 4 ? 3 : kSlots - 1;
    const bool listed = n_inst > 1 && n_inst <= kListMax;
    int* aoff = reinterpret_cast<int*>(bufs + bufs_bytes(nw, P.buf_rows));
    unsigned short* aidx = reinterpret_cast<unsigned short*>(aoff + n_inst + 1);
    int cur_b = -1;
    long long coef_item = -1;  // item whose next coefficients are in C.coef
    unsigned bar_target = 0;   // arrivals of the grid barriers so far
    if (threadIdx.x == 0) C.bad = 0;

    // prologue: pending status (KEQ_ERR_TIMEOUT until the statistics run) and
    // the items' first moments; residuals, counters and tickets are cleared by
    // the launch
    for (int b = blockIdx.x; b < n_inst; b += G) {
        const ImpInst& I = P.inst[b];
        if (threadIdx.x != 0 || !inst_enabled(I)) continue;
        I.stats->status = KEQ_ERR_TIMEOUT;
        if (P.head.fresh) {
            I.stats->total_iters = 0;
            I.stats->total_steps = 0;
        }
    }
    for (long long t = blockIdx.x; t < total_items; t += G) {
        __syncthreads();
        stage_inst(C, P, find_inst(P.item_off, n_inst, t), cur_b);
        if (!inst_enabled(C.I)) continue;
        first_item(C, wbuf, part, (int)(t - C.I.item_off), swap_io ? C.I.f_out : C.I.f_in,
                   swap_io ? const_cast<double*>(C.I.f_in) : C.I.f_out, smask);
        coef_item = t;
    }
    for (int m = -1; m < max_iter; ++m) {  // -1: the barrier behind the prologue
        if (m >= 0) {
            long long items = total_items;
            if (listed) {
                items = active_list(C, P, n_inst, m, aoff, aidx);
                if (items == 0) break;
            } else {
                bool some = false;
                for (int b = threadIdx.x; b < n_inst && !some; b += blockDim.x)
                    some = inst_active_rows(P.inst[b], m);
                if (!__syncthreads_or(some)) break;
            }
            const bool single = items <= (long long)G;  // every item has a CTA of its own
            if (traced) trace_mark(P, m, 0, true);
            int claim_par = 0;
            for (long long t = blockIdx.x; t < items;) {
                int blk;
                if (listed) {
                    int lo = 0, hi = C.n_act;  // aoff[lo] <= t < aoff[hi]
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (aoff[mid] <= (int)t) lo = mid; else hi = mid;
                    }
                    blk = (int)t - aoff[lo];
                    stage_inst(C, P, aidx[lo], cur_b);
                } else {
                    stage_inst(C, P, find_inst(P.item_off, n_inst, t), cur_b);
                    blk = (int)(t - C.I.item_off);
                }
                const ImpInst& I = C.I;
                const long long item = I.item_off + blk;
                if (listed || inst_active_rows(I, m)) {
                    const double* fn = swap_io ? I.f_out : I.f_in;
                    double* fo = swap_io ? const_cast<double*>(I.f_in) : I.f_out;
                    if (warp < I.nvt) copy_tile(I, wbuf, make_tile(I, blk, warp), fn);
                    if (warp == 0) stage_rows_coef<kAA>(C, blk, m, coef_item == item);
                    __syncthreads();
                    const double Gb = C.gbound, nm = C.nm;
                    PicardResidual pr(I.tol, I.abs_tol);
                    bool bad = false, ok = true;
                    for (int vt = warp; vt < I.nvt; vt += nw) {
                        const Tile g = make_tile(I, blk, vt);
                        ok &= I.conv_type == 0
                                  ? sweep_tile<true, 3>(C, wbuf, part[vt & smask], vt <= smask, g, blk, vt, m, I.dtdx, Gb, BarrierMaps{}, limit, fn, fo, pr, bad)
                                  : sweep_tile<false, 3>(C, wbuf, part[vt & smask], vt <= smask, g, blk, vt, m, I.dtdx, Gb, BarrierMaps{}, limit, fn, fo, pr, bad);
                        if (vt + nw < I.nvt) copy_tile(I, wbuf, make_tile(I, blk, vt + nw), fn);
                    }
                    if (!ok && lane == 0) {
                        atomicOr(&P.head.err, 1 << KEQ_ERR_TIMEOUT);
                        atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
                    }
                    if (I.conv_type == 0) {
                        double r1, r2;
                        pr.values(r1, r2);
                        r1 = warp_max_bits(r1);
                        r2 = warp_max_bits(r2);
                        if (lane == 0) {
                            C.red[warp][0] = r1;
                            C.red[warp][1] = r2;
                        }
                    }
                    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&C.bad, 1);
                    __syncthreads();
                    // the next item is claimed only now, with no wait of this one
                    // left: a CTA that held a claim while it waits could hold up
                    // the CTA it waits for
                    if (!single && threadIdx.x == kClaim) C.next[claim_par] = G + atomicAdd(&tickets[m], 1u);
                    if (warp == 0) finish_item<kAA>(C, buf0, part, blk, m, nm, smask);
                    if (warp == 1) flush_residuals(C, m);
                    coef_item = item;
                    if (kAA && aa_applies(I, m)) {
                        if (kThreads == 64) {
                            if (warp == 1)
                                for (int h = 0; h < 2; ++h) older_columns(C, buf0, blk, m, h);
                        } else if (warp == 2 || warp == 3) {
                            older_columns(C, buf0, blk, m, warp - 2);
                        }
                        __syncthreads();
                        gram_partials(C, buf0, blk, m);
                        __syncthreads();
                        // (beside the next item's coefficients: no barrier follows)
                        if (warp == nw - 1) {
                            unsigned prev = 0;
                            if (lane == 0) {
                                fence_acq_rel();
                                prev = atomicAdd(&I.rbdone[m], 1u);
                                fence_acq_rel();
                            }
                            prev = __shfl_sync(0xffffffffu, prev, 0);
                            if (prev == (unsigned)I.nblk - 1) last_block_alpha(C, m);
                        }
                        if (single) break;
                        t = C.next[claim_par];
                        claim_par ^= 1;
                        continue;
                    }
                } else if (!single && threadIdx.x == kClaim) {
                    C.next[claim_par] = G + atomicAdd(&tickets[m], 1u);
                }
                if (single) break;
                __syncthreads();
                t = C.next[claim_par];
                claim_par ^= 1;
            }
            if (traced) trace_mark(P, m, 1, false);
        }
        bar_target += G;
        __syncthreads();
        if (threadIdx.x == 0) {
            bar_arrive_nr(bar, 1u);
            C.ok = bar_wait(bar, bar_target, &P.head.err, limit) ? 1 : 0;
            if (!C.ok) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
        }
        __syncthreads();
        if (!C.ok) return;
    }

    // statistics
    if (blockIdx.x == 0 && threadIdx.x == 0) P.head.fresh = 0;
    for (int b = blockIdx.x; b < n_inst; b += G) {
        if (threadIdx.x >= 32) continue;
        const ImpInst& I = P.inst[b];
        if (!inst_enabled(I)) continue;
        int last;  // index of the last iteration that ran
        if (I.fixed_iters > 0) {
            last = (I.fixed_iters < I.picard_iter ? I.fixed_iters : I.picard_iter) - 1;
        } else {
            last = I.picard_iter - 1;
            for (int base = 0; base < I.picard_iter; base += 32) {
                const int q = base + lane;
                const bool stop = q < I.picard_iter && ld_cg(&I.res[2 * q]) <= 1.0;
                const unsigned mk = __ballot_sync(0xffffffffu, stop);
                if (mk != 0u) {
                    last = base + __ffs(mk) - 1;
                    break;
                }
            }
        }
        if (lane != 0) continue;
        int status = __ldcg(&I.nonfin[last]) ? KEQ_ERR_NONFINITE : KEQ_OK;
        if (__ldcg(&P.head.err) & (1 << KEQ_ERR_TIMEOUT)) status = KEQ_ERR_TIMEOUT;
        write_stats(I, last, status, ld_cg(&I.res[2 * last]), ld_cg(&I.res[2 * last + 1]));
    }
}

}  // namespace rows

const void* implicit_rows_entry(int threads, bool aa) {
    if (aa)
        return threads == 64    ? (const void*)rows::implicit_rows_kernel<64, 10, true>
               : threads == 128 ? (const void*)rows::implicit_rows_kernel<128, 5, true>
                                : (const void*)rows::implicit_rows_kernel<512, 1, true>;
    return threads == 64    ? (const void*)rows::implicit_rows_kernel<64, 10, false>
           : threads == 128 ? (const void*)rows::implicit_rows_kernel<128, 5, false>
                            : (const void*)rows::implicit_rows_kernel<512, 1, false>;
}
size_t implicit_rows_smem(int warps, int nslot, int n_inst, int buf_rows) {
    return sizeof(rows::CtaSmem) + (size_t)nslot * 3 * 32 * sizeof(double) +
           rows::bufs_bytes(warps, buf_rows) +
           (n_inst > 1 && n_inst <= rows::kListMax ? 6 * ((size_t)n_inst + 2) : 0);
}

}  // namespace keq
