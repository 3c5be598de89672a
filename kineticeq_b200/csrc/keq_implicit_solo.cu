// keq_implicit_solo.cu -- the implicit step of ONE instance with a CTA for
// every row block (a plan of one instance whose blocks are all resident).
// Sweep and results as in keq_implicit_rows.cu, bit for bit; what differs is
// how the CTAs of an iteration meet.
//
// There is no grid barrier.  A CTA publishes its block's maps, its residual
// maxima and its largest density as tagged words (each 64-bit word carries 32
// bits of a value and the iteration number) and reads those of all blocks.  A
// word is valid by itself, so nothing is fenced, counted or cleared between
// iterations, and one store-to-load latency replaces atomics, a release, the
// arrival count, its polling and the reload of the results: on one B200 4900 of
// the 15500 cycles of an iteration of 256x128.  Records alternate between two
// sets: a CTA overwrites a record of iteration m in iteration m+2, after it has
// read every block's record of m+1, and a block publishes that only once it is
// done with the records of m.  Behind the records of m no block reads maps of m
// any more, so one set of maps does where they are published behind them; the
// form that sweeps ahead (kAhead) has two.  The one barrier of a launch follows
// the prologue, which clears the tags of the launch before.
//
// The row update of a CTA stays in shared memory: W, the coefficients, the
// Anderson history; W goes to HBM at the end.  It starts when the row sums are
// there and does not wait for the residual quotients, which other warps form.
#include <cuda_runtime.h>

#include "keq_rows.cuh"

namespace keq {
namespace rows {

struct alignas(16) SoloSmem : BlockSmem {
    double W[3][32];               // W^(m) of the block's rows
    double red[kSlots][2];         // per warp: residual maxima
    double all[2][kSlots];         // per warp: residual maximum over the blocks read, by parity
    unsigned all_n[2][kSlots][2];  // the same: high word of the largest n, flags
    double g2[kMaxAACols][kMaxAACols];  // Gram matrix by ring column
    double wb[2][3];               // moments of the boundary rows
    double frac[6][32];            // warp 2's residual fractions
    double gbound;
    int bad[2];  // flags of the sweep (kBad...), by parity
    int set;     // set of PlanDev::maxima
};

// Anderson history of the block's rows: residual and moment columns.
struct Ring {
    double R[kMaxAACols][3][32], G[kMaxAACols][3][32];
};

constexpr int kRec = 4;  // 16-byte units of a block's record: residuals (2), n and flags (1), pad

// Gram matrix entries of two pairs from the blocks' tagged partials (one warp),
// summed in the order of aa_pair_sums.
__device__ __forceinline__ bool pair_sum2_tagged(const ulonglong2* ga, const ulonglong2* gb, int nblk,
                                                 unsigned tag, unsigned long long limit, double& va,
                                                 double& vb) {
    const int lane = threadIdx.x & 31;
    va = vb = 0.0;
    for (int r0 = 0; r0 < nblk; r0 += 160) {
        double t[5], u[5];
        unsigned long long it = 0;
        for (;;) {
            bool miss = false;
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const int r = r0 + 32 * c + lane < nblk ? r0 + 32 * c + lane : nblk - 1;
                miss |= !ld_tagged(ga + r, tag, t[c]);
                miss |= !ld_tagged(gb + r, tag, u[c]);
            }
            if (!__any_sync(0xffffffffu, miss)) break;
            if (++it > limit) return false;
        }
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const bool in = r0 + 32 * c + lane < nblk;
            va += in ? t[c] : 0.0;
            vb += in ? u[c] : 0.0;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        va += __shfl_xor_sync(0xffffffffu, va, o);
        vb += __shfl_xor_sync(0xffffffffu, vb, o);
    }
    return true;
}

// Ring columns of entry t of the Gram matrix of mh columns, oldest first from
// column col0: all pairs, or (all == false) the newest column with each.  The
// columns do not change once written, so a call that follows on another takes
// the older entries from there (28 pairs became 7).
__device__ __forceinline__ void gram_columns(const ImpInst& I, int t, int mh, int col0, bool all, int& cp,
                                             int& cq) {
    int p = t, q = mh - 1;
    if (all) aa_pair_of(t, mh, p, q);
    cp = col0 + p >= I.aa_cols ? col0 + p - I.aa_cols : col0 + p;
    cq = col0 + q >= I.aa_cols ? col0 + q - I.aa_cols : col0 + q;
}

// W^(m) after an applied Anderson call, by the whole CTA: every CTA sums the
// Gram partials of all blocks and solves the small system itself, which saves
// the round trips of one CTA doing it for all.  The sum of the |weights| plus
// one goes to C.gbound.
__device__ __noinline__ bool solo_combine(SoloSmem& C, const Ring* ring, const ulonglong2* gram, int m,
                                          int nr, bool all, unsigned long long limit) {
    const ImpInst& I = C.I;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int mh = m < I.aa_cols ? m : I.aa_cols;  // history of call m-1
    const int newest = (m - 1) % I.aa_cols;
    const int col0 = newest + 1 >= mh ? newest + 1 - mh : newest + 1 - mh + I.aa_cols;
    const int nsum = all ? mh * (mh + 1) / 2 : mh;
    auto put = [&](int t, double v) {
        int cp, cq;
        gram_columns(I, t, mh, col0, all, cp, cq);
        C.g2[cp][cq] = v;
        C.g2[cq][cp] = v;
    };
    const ulonglong2* gp = gram + (size_t)((m - 1) & 1) * kMaxPairs * I.nblk;
    bool ok = true;
    for (int t = warp; t < nsum; t += 2 * nw) {
        const int t2 = t + nw < nsum ? t + nw : t;  // two pairs in flight
        double v, v2;
        ok &= pair_sum2_tagged(gp + (size_t)t * I.nblk, gp + (size_t)t2 * I.nblk, I.nblk, (unsigned)m,
                               limit, v, v2);
        if (lane == 0) {
            put(t, v);
            put(t2, v2);
        }
    }
    __syncthreads();
    if (warp == 0) {
        const double al = aa_solve_gram(
            [&](int p, int q) {
                const int cp = col0 + p, cq = col0 + q;
                return C.g2[cp >= I.aa_cols ? cp - I.aa_cols : cp][cq >= I.aa_cols ? cq - I.aa_cols : cq];
            },
            mh, I.aa_reg, I.aa_alpha_max);
        int col = col0;
        double acc[3] = {0.0, 0.0, 0.0}, wnew[3], asum = 1.0;
        for (int jj = 0; jj < mh; ++jj) {
            const double aj = __shfl_sync(0xffffffffu, al, jj);
            asum += fabs(aj);
#pragma unroll
            for (int q = 0; q < 3; ++q) acc[q] = fma(ring->G[col][q][lane], aj, acc[q]);
            col = col + 1 == I.aa_cols ? 0 : col + 1;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) wnew[q] = ring->G[newest][q][lane];
        double w3[3], c4[4];
        combine_row(I, acc, wnew, w3, c4);
        if (lane < nr) {
#pragma unroll
            for (int q = 0; q < 3; ++q) C.W[q][lane] = w3[q];
            put_coef(C, lane, nr, c4);
        }
        if (lane == 0) C.gbound = asum;
    }
    __syncthreads();
    return ok;
}

// Row update at the end of a sweep (one warp, lane = row): moments of the new
// iterate, "w" residual, Anderson history, W and coefficients of the next
// iteration.  rec: the block's record.
template <bool kF, bool kAA>
__device__ __noinline__ void solo_update(SoloSmem& C, Ring* ring, const double (*part)[3][32], int blk,
                                         int m, int nr, ulonglong2* rec) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const bool ok = lane < nr;
    const double s0 = slot_sum<3>(part, I.nvt, 0);
    {  // largest density and the flags first: every block waits for them
        const double nb = n_bound(ok, s0 * I.dv);
        const int nan = any_nan_row(ok, s0 * I.dv) ? kBadNan : 0;
        if (lane == 0) {
            st_tagged(rec + 2, __hiloint2double(__double2hiint(nb), C.bad[m & 1] | nan), (unsigned)m + 1u);
            C.bad[(m & 1) ^ 1] = 0;
        }
    }
    const double s1 = slot_sum<3>(part, I.nvt, 1), s2 = slot_sum<3>(part, I.nvt, 2);
    double wn[3] = {0.0, 0.0, 0.0}, c4[4];
    if (ok) moments_and_coeffs(s0, s1, s2, I.dv, I.dt, I.tau_tilde, 1e-12, wn, c4);
    if (!kF) {
        FracMax q1, q2;
        if (ok) {
            const double wo[3] = {C.W[0][lane], C.W[1][lane], C.W[2][lane]};
            residual_w(wn, wo, I.abs_tol, I.tol, q1, q2);
        }
        if (blk == 0 && lane < 2) {  // the two boundary rows; their W is floored from iteration 1 on
            const double* b = C.wb[lane];
            const double o[3] = {m == 0 ? b[0] : clamp_min_t(b[0], 1e-12), b[1],
                                 m == 0 ? b[2] : clamp_min_t(b[2], 1e-12)};
            residual_w(b, o, I.abs_tol, I.tol, q1, q2);
        }
        const double r1 = warp_max(frac_value(q1)), r2 = warp_max(frac_value(q2));
        if (lane == 0) {
            st_tagged(rec, r1, (unsigned)m + 1u);
            st_tagged(rec + 1, r2, (unsigned)m + 1u);
        }
    }
    if (kAA) {
        const int head_in = m % I.aa_cols;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            ring->G[head_in][q][lane] = wn[q];
            ring->R[head_in][q][lane] = ok ? wn[q] - C.W[q][lane] : 0.0;
        }
        // the other warps form the Gram partials from here on (in front of the
        // residual, which every block waits for first: 1537x201 226 -> 256 us)
        __syncwarp();
        if (aa_applies(I, m)) asm volatile("bar.arrive 3, %0;" ::"r"(blockDim.x) : "memory");
    }
    if (ok && !(kAA && aa_applies(I, m))) {  // bgk1d_implicit_cuda_kernel.py:285-287
        C.W[0][lane] = clamp_min_t(wn[0], 1e-12);
        C.W[1][lane] = wn[1];
        C.W[2][lane] = clamp_min_t(wn[2], 1e-12);
        put_coef(C, lane, nr, c4);
    }
    __syncwarp();
}

// Gram partials of an applied Anderson call over the block's rows: a warp (all
// but warp 2, which updates the rows) per pair of columns, a lane per row.
__device__ __forceinline__ void solo_gram(const SoloSmem& C, const Ring* ring, ulonglong2* gram, int blk,
                                          int m, bool all) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31, nw = (blockDim.x >> 5) - 1;
    const int warp = threadIdx.x >> 5 < 2 ? threadIdx.x >> 5 : (threadIdx.x >> 5) - 1;  // without warp 2
    const int cols = I.aa_cols;
    const int mh = (m + 1) < cols ? (m + 1) : cols;
    const int newest = m % cols;
    const int col0 = newest + 1 >= mh ? newest + 1 - mh : newest + 1 - mh + cols;
    const int nsum = all ? mh * (mh + 1) / 2 : mh;
    ulonglong2* gp = gram + (size_t)(m & 1) * kMaxPairs * I.nblk;
    for (int t = warp; t < nsum; t += nw) {
        int cp, cq;
        gram_columns(I, t, mh, col0, all, cp, cq);
        double v = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) v = fma(ring->R[cp][c][lane], ring->R[cq][c][lane], v);
        v = warp_sum(v);
        if (lane == 0) st_tagged(gp + (size_t)t * I.nblk + blk, v, (unsigned)m + 1u);
    }
}

// kF: convergence on f (else on the moments); kAA: Anderson.  A kernel for each:
// one that holds all of it spills and misses the instruction cache (256x128 64.1
// us a step against 60.8, 4096x512 195.4 against 189.5).
//
// kAhead: the first half of the sweep of iteration m+1 goes ahead of the test
// whether there is to be one: it needs the block's own rows only and writes
// nothing but maps, and the records of iteration m arrive meanwhile.  256x128
// 61.4 -> 54.2 us a step, 124x64 36.4 -> 33.3, 4096x64 116 -> 90, 8192x128 138 ->
// 108, 700x200 83 -> 76, 8192x256 192 -> 164.  For CTAs of up to eight warps with
// a tile each: with 16 warps the barrier behind the first halves keeps one
// warp's arithmetic from overlapping another's memory
// traffic (4096x512 189 -> 200, and 225 when every warp reads the records by
// itself instead).  After an applied Anderson call the sweep needs the exchange.
template <bool kF, bool kAA, bool kAhead>
__global__ void __launch_bounds__(kAhead ? 256 : 512, kAhead ? 2 : 1)
implicit_solo_kernel(PlanDev* __restrict__ Pp, int swap_io) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlanDev& P = *Pp;
    SoloSmem& C = *reinterpret_cast<SoloSmem*>(smem_raw);
    const ImpInst& I = C.I;
    const unsigned long long limit = P.head.spin_limit;
    const bool traced = P.head.trace != nullptr;
    const int nslot = P.nslot;
    ulonglong2* const gather = P.gather;
    ulonglong2* const gram = P.gram;
    double(*part)[3][32] = reinterpret_cast<double(*)[3][32]>(smem_raw + sizeof(SoloSmem));
    TileBuf* bufs = reinterpret_cast<TileBuf*>(part + nslot);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const int blk = (int)blockIdx.x;
    {
        const int* s = reinterpret_cast<const int*>(&P.inst[0]);
        int* d = reinterpret_cast<int*>(&C.I);
        for (int q = tid; q < (int)(sizeof(ImpInst) / sizeof(int)); q += blockDim.x) d[q] = __ldg(s + q);
        if (tid == 0) {
            C.bad[0] = C.bad[1] = 0;
            C.set = launch_parity(&P.arrivals, gridDim.x);
        }
    }
    __syncthreads();
    double* const maxima = P.maxima[C.set];
    if (!inst_enabled(I)) {
        if (blk == 0 && tid == 0) P.head.fresh = 0;
        return;
    }
    // one set of maps, but two where they go out ahead of the records (kAhead)
    ulonglong2* const set0 = reinterpret_cast<ulonglong2*>(I.xch);
    TaggedMaps maps{{set0, kAhead ? P.maps : set0}, 0u, nullptr, 0};
    Ring* const ring = kAA ? reinterpret_cast<Ring*>(bufs + nw) : nullptr;
    const double* fn = swap_io ? I.f_out : I.f_in;
    double* fo = swap_io ? const_cast<double*>(I.f_in) : I.f_out;
    const int nr = I.n_inner - blk * I.rblk < I.rblk ? I.n_inner - blk * I.rblk : I.rblk;

    // prologue: pending status (KEQ_ERR_TIMEOUT until the statistics are
    // written), tags of the launch before, moments of f^n and W^(0)
    if (blk == 0 && tid < kMaxima) P.maxima[C.set ^ 1][tid] = 0.0;
    if (blk == 0 && tid == 0) {
        I.stats->status = KEQ_ERR_TIMEOUT;
        if (P.head.fresh) {
            I.stats->total_iters = 0;
            I.stats->total_steps = 0;
        }
    }
    for (int vt = warp; vt < I.nvt; vt += nw)
#pragma unroll
        for (int par = 0; par < (kAhead ? 2 : 1); ++par) {
            ulonglong2* p = maps.slot(I, par, blk, vt);
            st_tagged(p, 0.0, 0u);
            st_tagged(p + 32, 0.0, 0u);
        }
    if (tid < 2 * kRec)
        st_tagged(gather + ((size_t)(tid / kRec) * I.nblk + blk) * kRec + tid % kRec, 0.0, 0u);
    if (kAA)
        for (int t = tid; t < 2 * kMaxPairs; t += blockDim.x)
            st_tagged(gram + (size_t)t * I.nblk + blk, 0.0, 0u);
    {
        double mx = warp_max_bits(first_tiles(C, bufs[warp], part, blk, fn, fo));
        if (lane == 0) C.red[warp][0] = mx;
        __syncthreads();
        if (warp == 0) {
            mx = warp_max_bits(lane < nw ? C.red[lane][0] : 0.0);
            double w3[3] = {0.0, 0.0, 0.0}, c4[4] = {0.0, 0.0, 0.0, 0.0};
            const double s0 = slot_sum<3>(part, I.nvt, 0);
            if (lane < nr) {
                moments_and_coeffs(s0, slot_sum<3>(part, I.nvt, 1), slot_sum<3>(part, I.nvt, 2), I.dv, I.dt, I.tau_tilde, 0.0, w3, c4);
#pragma unroll
                for (int q = 0; q < 3; ++q) C.W[q][lane] = w3[q];
                put_coef(C, lane, nr, c4);
            }
            const double n = warp_max_bits(w3[0]), cm = warp_max_bits(c4[2]);
            if (any_nan_row(lane < nr, s0 * I.dv) && lane == 0) {
                atomic_max_nonneg(&maxima[3], (double)(blk + 1));
                atomic_max_nonneg(&maxima[4], (double)(I.nblk - blk));
            }
            if (lane == 0) {
                atomic_max_nonneg(&maxima[0], mx);
                atomic_max_nonneg(&maxima[1], cm);
                atomic_max_nonneg(&maxima[2], n);
            }
        }
    }
    if (!launch_barrier(&P.arrivals, gridDim.x, limit)) {
        if (tid == 0) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
        return;
    }
    const double fmx = ld_cg(&maxima[0]), cm0 = ld_cg(&maxima[1]);
    double nm = ld_cg(&maxima[2]);
    // blocks with NaN rows upstream of this one: of v > 0 (bit 0), of v <= 0 (bit 1)
    int nan_in = (I.nblk - ld_cg(&maxima[4]) < blk ? 1 : 0) | (ld_cg(&maxima[3]) - 1.0 > blk ? 2 : 0);
    if (!kF && tid < 6) C.wb[tid / 3][tid % 3] = ld_cg(&I.Wb[tid]);
    if (warp < I.nvt) copy_tile(I, bufs[warp], make_tile(I, blk, warp), fn);

    // iterations at most; a replay runs exactly this many
    const int iter_max = I.fixed_iters > 0 && I.fixed_iters < I.picard_iter ? I.fixed_iters : I.picard_iter;
    double std_res = 0.0;
    bool bad_last = false, failed = false;
    int gram_m = -2;  // last iteration with a Gram matrix
    bool gram_all = true;
    int m = 0;  // in the end the number of iterations
    bool ok = true;
    for (;; ++m) {
        const unsigned tag = (unsigned)m + 1u;
        maps.tag = tag;
        double asum = 1.0;
        const bool more = m < iter_max;
        SweepState<TaggedMaps> S;
        Tile g0;
        if (kAhead && warp < I.nvt) {
            S.maps = maps;
            g0 = make_tile(I, blk, warp);
            if (more) sweep_begin(C, bufs[warp], g0, blk, warp, m, I.dtdx, fn, S);
        }
        if (m > 0) {
            const int par = (m - 1) & 1;
            const ulonglong2* recs = gather + (size_t)par * I.nblk * kRec;
            double a1 = 0.0;
            unsigned an = 0u, ab = 0u;
            // (in front of the sweep: the warps without a part in the row update first)
            int t0 = kAhead ? tid : tid - 96;
            if (t0 < 0) t0 += blockDim.x;
            for (int t = t0; t < I.nblk; t += blockDim.x) {
                const ulonglong2* p = recs + (size_t)t * kRec;
                double r1, nb;
                unsigned long long it = 0;
                for (;;) {
                    bool there = ld_tagged(p, tag - 1u, r1);
                    there &= ld_tagged(p + 2, tag - 1u, nb);
                    if (there) break;
                    if (++it > limit) {
                        ok = false;
                        break;
                    }
                }
                // non-negative values and +NaN order like their bits
                a1 = __double_as_longlong(r1) > __double_as_longlong(a1) ? r1 : a1;
                const unsigned h = (unsigned)__double2hiint(nb);
                an = h > an ? h : an;
                ab |= (unsigned)__double2loint(nb);
            }
            __syncwarp();
            a1 = warp_max_bits(a1);
            an = __reduce_max_sync(0xffffffffu, an);
            ab = __reduce_or_sync(0xffffffffu, ab);
            if (lane == 0) {
                C.all[par][warp] = a1;
                C.all_n[par][warp][0] = an;
                C.all_n[par][warp][1] = ab;
            }
            if (!__syncthreads_and(ok)) {
                failed = true;
                break;
            }
            std_res = warp_max_bits(lane < nw ? C.all[par][lane] : 0.0);
            const unsigned hn = __reduce_max_sync(0xffffffffu, lane < nw ? C.all_n[par][lane][0] : 0u);
            bad_last = false;
            nan_in = 0;
            if (__any_sync(0xffffffffu, lane < nw && C.all_n[par][lane][1] != 0u)) {
                const unsigned flags = __reduce_or_sync(0xffffffffu, lane < nw ? C.all_n[par][lane][1] : 0u);
                bad_last = (flags & kBadValue) != 0u;
                failed = (flags & kBadWait) != 0u;
                // the blocks with NaNs, from the records once more (they are there)
                for (int t = lane; t < I.nblk && (flags & kBadNan); t += 32) {
                    double nb;
                    const bool there = ld_tagged(recs + (size_t)t * kRec + 2, tag - 1u, nb);
                    if (there && ((unsigned)__double2loint(nb) & kBadNan)) nan_in |= t < blk ? 1 : (t > blk ? 2 : 0);
                }
                __syncwarp();
                nan_in = (int)__reduce_or_sync(0xffffffffu, (unsigned)nan_in);
                if (failed) break;
            }
            const double nb = __hiloint2double((int)hn, -1);
            nm = nb > nm ? nb : nm;
            if (!more || (I.fixed_iters <= 0 && std_res <= 1.0)) break;
        }
        if (kAA && m >= 1 && aa_applies(I, m - 1)) {
            ok = solo_combine(C, ring, gram, m, nr, gram_all, limit);
            asum = C.gbound;
        }
        if (!kAhead && nan_in != 0) {
            if (tid < 2 && (nan_in >> tid & 1)) nan_inflow(C, tid);
            __syncthreads();
        }
        ulonglong2* rec = gather + ((size_t)(m & 1) * I.nblk + blk) * kRec;
        const double G = fold_bound(fmx, cm0, nm, m, asum);
        if (traced) trace_mark(P, m, 0, true);
        PicardResidual pr(I.tol, I.abs_tol);
        bool bad = false;
        if (kAhead) {
            if (warp < I.nvt) {
                if (nan_in & (g0.pos ? 1 : 2)) nan_inflow(S);
                ok &= sweep_end<kF, 3>(C, bufs[warp], part[warp], true, g0, blk, warp, m, I.dtdx, G, S, limit, fn,
                                       fo, pr, bad);
            }
        } else {
            for (int vt = warp; vt < I.nvt; vt += nw) {
                const Tile g = make_tile(I, blk, vt);
                ok &= sweep_tile<kF, 3>(C, bufs[warp], part[vt & (kSlots - 1)], vt < kSlots, g, blk, vt, m, I.dtdx,
                                        G, maps, limit, fn, fo, pr, bad);
                if (vt + nw < I.nvt) copy_tile(I, bufs[warp], make_tile(I, blk, vt + nw), fn);
            }
        }
        if (__any_sync(0xffffffffu, bad || !ok)) {
            const int flags = (__any_sync(0xffffffffu, bad) ? kBadValue : 0) | (__any_sync(0xffffffffu, !ok) ? kBadWait : 0);
            if (lane == 0) atomicOr(&C.bad[m & 1], flags);
        }
        if (traced) trace_mark(P, m, 1, false);
        // Warp 2 updates the rows as soon as all row sums are there (barrier 1);
        // warp 3 takes its residual fractions along.  The others meet once more
        // behind the residual quotients (barrier 2).
        if (warp == 2) {
            C.frac[0][lane] = pr.q1.num; C.frac[1][lane] = pr.q1.den; C.frac[2][lane] = pr.q1.special;
            C.frac[3][lane] = pr.q2.num; C.frac[4][lane] = pr.q2.den; C.frac[5][lane] = pr.q2.special;
        }
        if (warp == 2 || warp == 3)
            asm volatile("bar.sync 1, %0;" ::"r"(blockDim.x) : "memory");
        else
            asm volatile("bar.arrive 1, %0;" ::"r"(blockDim.x) : "memory");
        if (warp != 2) {
            if (kF) {
                if (warp == 3) {
                    larger(pr.q1.num, pr.q1.den, C.frac[0][lane], C.frac[1][lane]);
                    larger(pr.q2.num, pr.q2.den, C.frac[3][lane], C.frac[4][lane]);
                    const double s1 = C.frac[2][lane], s2 = C.frac[5][lane];  // >= 0 or +NaN
                    if (__double_as_longlong(s1) > __double_as_longlong(pr.q1.special)) pr.q1.special = s1;
                    if (__double_as_longlong(s2) > __double_as_longlong(pr.q2.special)) pr.q2.special = s2;
                }
                double r1, r2;
                pr.values(r1, r2);
                r1 = warp_max_bits(r1);
                r2 = warp_max_bits(r2);
                if (lane == 0) {
                    C.red[warp][0] = r1;
                    C.red[warp][1] = r2;
                }
            }
            asm volatile("bar.sync 2, %0;" ::"r"(blockDim.x - 32) : "memory");
        }
        if (warp == 1) {
            if (kF) {
                const double r1 = warp_max_bits(lane < nw && lane != 2 ? C.red[lane][0] : 0.0);
                const double r2 = warp_max_bits(lane < nw && lane != 2 ? C.red[lane][1] : 0.0);
                if (lane == 0) {
                    st_tagged(rec, r1, tag);
                    st_tagged(rec + 1, r2, tag);
                }
            }
        } else if (warp == 2) {
            solo_update<kF, kAA>(C, ring, part, blk, m, nr, rec);
        }
        if (kAA && aa_applies(I, m)) {
            gram_all = gram_m != m - 1;  // columns without entries besides the newest
            gram_m = m;
            if (warp != 2) {  // behind the history's newest column (solo_update)
                asm volatile("bar.sync 3, %0;" ::"r"(blockDim.x) : "memory");
                solo_gram(C, ring, gram, blk, m, gram_all);
            }
        }
        // next iteration's f^n (the copies of a CTA take the load unit for 2000
        // cycles: in front of a barrier they hold up the row update)
        if (warp < I.nvt) copy_tile(I, bufs[warp], make_tile(I, blk, warp), fn);
        if (kAhead && !__syncthreads_and(ok)) {  // the coefficients of the next iteration
            failed = true;
            break;
        }
    }
    cp_async_wait_all();
    if (failed) {
        if (tid == 0) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
        return;
    }
    if (warp == 0 && lane < nr) {
        const int i = blk * I.rblk + lane + 1;
#pragma unroll
        for (int q = 0; q < 3; ++q) I.W[(size_t)q * I.nx + i] = C.W[q][lane];
    }
    if (blk == 0 && warp == 1 && lane < 2) {  // floored moments of the fixed rows
        const int ib = lane == 0 ? 0 : I.nx - 1;
        I.W[ib] = clamp_min_t(ld_cg(&I.Wb[3 * lane + 0]), 1e-12);
        I.W[I.nx + ib] = ld_cg(&I.Wb[3 * lane + 1]);
        I.W[2 * (size_t)I.nx + ib] = clamp_min_t(ld_cg(&I.Wb[3 * lane + 2]), 1e-12);
    }
    if (blk == 0 && warp == 0) {
        // the relative residual of the last iteration is read once, for the statistics
        double res = 0.0;
        for (int t = lane; t < I.nblk; t += 32) {
            const ulonglong2* p = gather + ((size_t)((m - 1) & 1) * I.nblk + t) * kRec + 1;
            double r2;
            unsigned long long it = 0;
            while (!ld_tagged(p, (unsigned)m, r2))
                if (++it > limit) {
                    ok = false;
                    break;
                }
            res = __double_as_longlong(r2) > __double_as_longlong(res) ? r2 : res;
        }
        __syncwarp();
        res = warp_max_bits(res);
        if (!__all_sync(0xffffffffu, ok)) {  // the pending status stays
            if (lane == 0) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
        } else if (lane == 0) {
            P.head.fresh = 0;
            write_stats(I, m - 1, bad_last ? KEQ_ERR_NONFINITE : KEQ_OK, std_res, res);
        }
    }
}

}  // namespace rows

// ahead: one tile per warp at most and few warps (see kAhead).
const void* implicit_solo_entry(int conv_type, int aa_on, bool ahead) {
    if (aa_on)
        return conv_type == 0 ? (const void*)rows::implicit_solo_kernel<true, true, false>
                              : (const void*)rows::implicit_solo_kernel<false, true, false>;
    if (ahead)
        return conv_type == 0 ? (const void*)rows::implicit_solo_kernel<true, false, true>
                              : (const void*)rows::implicit_solo_kernel<false, false, true>;
    return conv_type == 0 ? (const void*)rows::implicit_solo_kernel<true, false, false>
                          : (const void*)rows::implicit_solo_kernel<false, false, false>;
}
size_t implicit_solo_smem(int warps, int nslot, int ring) {
    return sizeof(rows::SoloSmem) + (size_t)nslot * 3 * 32 * sizeof(double) +
           (size_t)warps * sizeof(rows::TileBuf) + (ring ? sizeof(rows::Ring) : 0);
}
size_t implicit_solo_gather_units(int nblk) { return 2 * (size_t)nblk * rows::kRec; }

}  // namespace keq
