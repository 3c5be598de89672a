// keq_gtsv.cu -- batched tridiagonal solve behind keq_gtsv_strided_inplace and
// keq_gtsv_strided_inplace_noalloc.
//
// One CTA per system of 16 rows or more (a thread per smaller system).  A system
// whose rows are all strictly diagonally dominant (every system of the implicit
// schemes is) is solved by the partition method: a thread owns L consecutive
// rows, eliminates all but the last of them from both ends, the last rows form a
// system of one unknown per thread that is solved by parallel cyclic reduction,
// and each thread then solves its rows between two known values.  Strict
// dominance carries over to every system on the way, so no pivot can vanish.  Any
// other system is solved by one thread with the Thomas algorithm of the
// reference's CPU twin (gtsv_cpu/gtsv_binding.cpp:32-37, 51-97: no pivoting,
// pivots floored to +-1e-300), operation for operation; so is one with a diagonal
// outside [1e-250, 1e250] or a right-hand side beyond 1e300, infinities and NaN
// included, which the reduction would keep to a few chunks.
//
// What bounds it: latency.  One thread per system, the algorithm of the CPU
// twin on the GPU, walked 2n dependent steps of an uncoalesced load and a
// division each (256 systems of 2046 rows: 1.87 ms on one B200 with 2 of 148
// SMs in use).  Here a system takes 2L steps plus the reduction, its rows are
// staged through shared memory with coalesced copies, and all SMs work: 12 us.
// L is odd, so that the strided accesses of neighbouring threads fall into
// different banks, and 9 where the thread count allows: shorter chunks move the
// work into the reduction, longer ones lengthen the chain.
#include <cuda_runtime.h>

#include "keq_common.cuh"
#include "keq_internal.h"

namespace keq {
namespace {

constexpr int kMaxT = 512;
constexpr size_t kSmemMax = 224 * 1024;

// One system by the Thomas algorithm, the modified diagonal in pi.
__device__ __forceinline__ void thomas(const double* pa, const double* pd, const double* pc, double* pr,
                                       double* pi, int n) {
    auto piv = [](double x) {
        if (fabs(x) >= 1.0e-300) return x;
        return x < 0.0 ? -1.0e-300 : 1.0e-300;
    };
    double dprev = pd[0];
    pi[0] = dprev;
    for (int i = 1; i < n; ++i) {
        const double w = pa[i] / piv(dprev);
        const double di = pd[i] - w * pc[i - 1];
        pr[i] -= w * pr[i - 1];
        pi[i] = di;
        dprev = di;
    }
    pr[n - 1] /= piv(pi[n - 1]);
    for (int i = n - 1; i-- > 0;) pr[i] = (pr[i] - pc[i] * pr[i + 1]) / piv(pi[i]);
}

// Rows in shared memory (kSmem) or in place, with cp (n per system) for the
// reciprocal pivots.
template <bool kSmem>
__global__ void __launch_bounds__(kMaxT) gtsv_kernel(const double* __restrict__ dl,
                                                     const double* __restrict__ d,
                                                     const double* __restrict__ du,
                                                     double* __restrict__ B, int n, int L,
                                                     double* __restrict__ cp, int defer) {
    extern __shared__ __align__(16) double sm[];
    const int T = blockDim.x, k = threadIdx.x;
    const size_t o = (size_t)blockIdx.x * n;
    double* ex = kSmem ? sm + 4 * (size_t)n : sm;  // exchange: 4 arrays of T
    const double* pa = kSmem ? sm : dl + o;
    const double* pd = kSmem ? sm + n : d + o;
    const double* pc = kSmem ? sm + 2 * (size_t)n : du + o;
    double* pr = kSmem ? sm + 3 * (size_t)n : B + o;
    double* pi = kSmem ? sm + n : cp + o;  // reciprocal pivots (over the diagonal in shared memory)
    if (kSmem) {
        for (int i = k; i < n; i += T) {
            cp_async8(sm + i, dl + o + i);
            cp_async8(sm + n + i, d + o + i);
            cp_async8(sm + 2 * (size_t)n + i, du + o + i);
            cp_async8(sm + 3 * (size_t)n + i, B + o + i);
        }
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
    }
    bool dom = true;
    for (int i = k; i < n; i += T) {
        const double a = i > 0 ? fabs(pa[i]) : 0.0, c = i < n - 1 ? fabs(pc[i]) : 0.0;
        const double b = fabs(pd[i]);
        dom &= b > a + c && b >= 1e-250 && b <= 1e250 && fabs(pr[i]) <= 1e300;
    }
    dom = __syncthreads_and(dom);
    if (kSmem && defer) {  // the other systems are gtsv_thread_kernel's
        if (k == 0) cp[o] = dom ? 0.0 : 1.0;
        if (!dom) return;
    }
    if (!dom) {
        if (k == 0) thomas(pa, pd, pc, pr, pi, n);
    } else {
        const int K = (n + L - 1) / L;
        const bool on = k < K;
        const int s = k * L, e = (s + L < n ? s + L : n) - 1;
        // the rows before the chunk's last, from both ends:
        //   x_{e-1} = y1 + P1 xi_{k-1} + Q1 xi_k,   x_s = y0 + P0 xi_{k-1} + Q0 xi_k
        double y0 = 0.0, P0 = 0.0, Q0 = 1.0, y1 = 0.0, P1 = 1.0, Q1 = 0.0;
        if (on && e > s) {
            double bi = 0.0, r = 0.0, p = 0.0, b2i = 0.0, r2 = 0.0, q2 = 0.0;
            for (int j = 0; j < e - s; ++j) {
                const int i = s + j, i2 = e - 1 - j;
                double b = pd[i], b2 = pd[i2];
                const double ri = pr[i], ri2 = pr[i2];
                if (j == 0) {
                    r = ri;
                    p = i > 0 ? -pa[i] : 0.0;
                    r2 = ri2;
                    q2 = -pc[i2];
                } else {
                    const double w = pa[i] * bi, w2 = pc[i2] * b2i;
                    b = fma(-w, pc[i - 1], b);
                    r = fma(-w, r, ri);
                    p = -w * p;
                    b2 = fma(-w2, pa[i2 + 1], b2);
                    r2 = fma(-w2, r2, ri2);
                    q2 = -w2 * q2;
                }
                bi = recip3(b);
                b2i = recip3(b2);
            }
            y1 = bi * r;
            P1 = bi * p;
            Q1 = -bi * pc[e - 1];
            y0 = b2i * r2;
            Q0 = b2i * q2;
            P0 = s > 0 ? -b2i * pa[s] : 0.0;
        }
        ex[k] = y0;
        ex[T + k] = P0;
        ex[2 * T + k] = Q0;
        __syncthreads();
        double al = 0.0, be = 1.0, ga = 0.0, de = 0.0;
        if (on) {
            const double a = e > 0 ? pa[e] : 0.0, c = e < n - 1 ? pc[e] : 0.0;
            const bool nx = k + 1 < K;
            const double yn = nx ? ex[k + 1] : 0.0, Pn = nx ? ex[T + k + 1] : 0.0,
                         Qn = nx ? ex[2 * T + k + 1] : 0.0;
            al = a * P1;
            be = fma(c, Pn, fma(a, Q1, pd[e]));
            ga = c * Qn;
            de = fma(-c, yn, fma(-a, y1, pr[e]));
        }
        // Parallel cyclic reduction.  It ends once the rows are decoupled to below
        // double rounding of the largest value (2^-60) and, entry by entry, the coupling
        // to the neighbours' values is small against the row's own (the Jacobi iteration
        // scaled by them contracts by 2^-58), or vanishes in a double's range: where a
        // solution decays, a value may be far below 2^-60 of its neighbours and consist
        // of what the coupling brings.  Couplings are squared at each step, so going on
        // to 1e-270 always would take four more (assembly and solve of 624 systems of
        // 4268 rows: 83 us a pass to 2^-60 alone, 92 to 1e-270, 86 with the comparison).
        for (int st = 1; st < K; st <<= 1) {
            const double rb = recip3(be);
            const double cpl = fabs(rb) * (fabs(al) + fabs(ga));
            if (__syncthreads_and(cpl <= 8.673617379884035e-19)) {  // (also: the reads of the step before are done)
                const double xh = fabs(de * rb);
                ex[k] = xh;
                __syncthreads();
                double g = 0.0;
                if (k >= st) g = fabs(al) * ex[k - st];
                if (k + st < K) g = fma(fabs(ga), ex[k + st], g);
                if (__syncthreads_and(fabs(rb) * g <= 3.469446951953614e-18 * xh || cpl <= 1e-270)) break;
            }
            ex[k] = al;
            ex[T + k] = rb;
            ex[2 * T + k] = ga;
            ex[3 * T + k] = de;
            __syncthreads();
            const bool lo = k >= st, hi = k + st < K;
            const int kl = lo ? k - st : k, kh = hi ? k + st : k;
            const double e1 = lo ? al * ex[T + kl] : 0.0, e2 = hi && on ? ga * ex[T + kh] : 0.0;
            be = fma(-e1, ex[2 * T + kl], fma(-e2, ex[kh], be));
            de = fma(-e1, ex[3 * T + kl], fma(-e2, ex[3 * T + kh], de));
            al = -e1 * ex[kl];
            ga = -e2 * ex[2 * T + kh];
        }
        const double xi = de * recip3(be);
        __syncthreads();
        ex[k] = xi;
        __syncthreads();
        if (on) {
            // the chunk between xi_{k-1} and xi_k
            double bi = 0.0, r = 0.0;
            for (int i = s; i < e; ++i) {
                double b = pd[i];
                if (i == s) {
                    r = s > 0 ? fma(-pa[s], ex[k - 1], pr[s]) : pr[s];
                } else {
                    const double w = pa[i] * bi;
                    b = fma(-w, pc[i - 1], b);
                    r = fma(-w, r, pr[i]);
                }
                bi = recip3(b);
                pi[i] = bi;
                pr[i] = r;
            }
            double x = xi;
            pr[e] = xi;
            for (int i = e - 1; i >= s; --i) {
                x = fma(-pc[i], x, pr[i]) * pi[i];
                pr[i] = x;
            }
        }
    }
    if (kSmem) {
        __syncthreads();
        for (int i = k; i < n; i += T) B[o + i] = pr[i];
    }
}

// A thread per system, by the same sequential algorithm, for
//  - systems of less than two chunks, and of less than three where there are many:
//    the partition saves few steps there, and a CTA of 32 threads each, of which one
//    to three work, costs more the more systems there are.  us per call, a CTA and a
//    thread per system: 262144 systems of 1 row 140 and 16, of 8 rows 216 and 56, of
//    15 rows 224 and 158; 65536 of 16 rows 60 and 58, of 20 rows 62 and 46, of 22
//    rows 60 and 50, of 24 rows 60 and 67; 8192 of 16 to 22 rows 13 and 15.  Bound by
//    the strided reads;
//  - the systems that are not dominant (cp[0] of a system says so) where there are
//    too many for one thread of a CTA each (kDeferWaves).
constexpr int kThreadRows = 15, kThreadRowsMany = 23, kMany = 32768;
__global__ void __launch_bounds__(128) gtsv_thread_kernel(const double* __restrict__ dl,
                                                          const double* __restrict__ d,
                                                          const double* __restrict__ du,
                                                          double* __restrict__ B, int n, int batch,
                                                          double* __restrict__ cp, int flagged) {
    if (flagged) cudaGridDependencySynchronize();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= batch) return;
    const size_t o = (size_t)b * n;
    if (flagged && cp[o] == 0.0) return;
    thomas(dl + o, d + o, du + o, B + o, cp + o, n);
}

// A CTA solves a system that is not dominant with one thread, from shared memory,
// about 2.7 times as fast as a thread of gtsv_thread_kernel does; that one has 128
// times the threads.  Waves of resident CTAs from which it wins.  us per call for
// systems that are not dominant, in the CTA and deferred: 8192 of 512 rows 1309 and
// 559, 65536 of 64 rows 361 and 264, 800 of 5000 rows 9963 and 5003; 1024 of 512 rows
// 226 and 547.  Dominant systems pay the second launch: 8192 of 512 rows 47 and 50, 800
// of 5000 rows 58 and 62 (63 and 64 without the early dispatch).
constexpr int kDeferWaves = 4;

}  // namespace

cudaError_t launch_gtsv(const double* dl, const double* d, const double* du, double* B, int n,
                        int batch, double* scratch, cudaStream_t s) {
    const int thread_blocks = (int)(((long long)batch + 127) / 128);
    if (n <= kThreadRows || (n <= kThreadRowsMany && batch >= kMany)) {
        gtsv_thread_kernel<<<thread_blocks, 128, 0, s>>>(dl, d, du, B, n, batch, scratch, 0);
        return cudaGetLastError();
    }
    // one warp up to 288 rows (chunks of 3 to 9), then chunks of 9 up to 4608
    // rows, then 512 threads
    int L = n <= 288 ? (n + 31) / 32 : (n <= 9 * kMaxT ? 9 : (n + kMaxT - 1) / kMaxT);
    L = L < 3 ? 3 : L | 1;
    const int T = ((n + L - 1) / L + 31) / 32 * 32;
    const size_t ex = 4 * (size_t)T * sizeof(double);
    const size_t full = ex + 4 * (size_t)n * sizeof(double);
    if (full <= kSmemMax) {
        if (full > 48 * 1024) {
            const cudaError_t e = cudaFuncSetAttribute(
                gtsv_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
            if (e != cudaSuccess) return e;
        }
        // CTAs resident on 148 SMs, by shared memory (1 KB of it is the system's) and
        // by threads
        const int by_smem = (int)(kSmemMax / (full + 1024)), by_threads = 2048 / T;
        const int occ = by_smem < by_threads ? by_smem : by_threads;
        const int defer = batch > (kDeferWaves - 1) * 148 * (occ < 1 ? 1 : occ < 32 ? occ : 32);
        gtsv_kernel<true><<<batch, T, full, s>>>(dl, d, du, B, n, L, scratch, defer);
        if (defer) {
            // dispatched as the first kernel drains; it waits for that one's stores
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at.val.programmaticStreamSerializationAllowed = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(thread_blocks);
            cfg.blockDim = dim3(128);
            cfg.stream = s;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            const cudaError_t e =
                cudaLaunchKernelEx(&cfg, gtsv_thread_kernel, dl, d, du, B, n, batch, scratch, 1);
            if (e != cudaSuccess) return e;
        }
    } else {
        gtsv_kernel<false><<<batch, T, ex, s>>>(dl, d, du, B, n, L, scratch, 0);
    }
    return cudaGetLastError();
}

}  // namespace keq
