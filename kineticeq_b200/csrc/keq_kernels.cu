// keq_kernels.cu -- kernel-level drop-ins of the reference's extension
// modules (implicit_fused, gtsv, lo_blocktridiag) behind the C ABI.  The
// fused time-step kernels (keq_implicit.cu, keq_holo.cu) do not call these;
// they serve callers that use the reference's module-level API directly.
#include <cuda_runtime.h>
#include <math.h>

#include "keq_common.cuh"
#include "keq_internal.h"
#include "keq_rows.cuh"

namespace keq {

// ---- K1: velocity moments, one warp per row -------------------------------
// implicit_kernels.cu:28-81 semantics (clamps), reduction = per-lane strided
// partial sums + fixed butterfly.
__global__ void __launch_bounds__(256) moments_kernel(const double* __restrict__ f,
                                                      const double* __restrict__ v, int nx,
                                                      int nv, double dv, double* __restrict__ n,
                                                      double* __restrict__ nu,
                                                      double* __restrict__ T) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= nx) return;
    const double* row = f + (size_t)warp * nv;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    for (int j = lane; j < nv; j += 32) {
        const double x = row[j], vj = v[j];
        p0 += x;
        p1 += x * vj;
        p2 += x * vj * vj;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        p0 += __shfl_xor_sync(0xffffffffu, p0, o);
        p1 += __shfl_xor_sync(0xffffffffu, p1, o);
        p2 += __shfl_xor_sync(0xffffffffu, p2, o);
    }
    if (lane == 0) {
        const double n_raw = p0 * dv, nu_raw = p1 * dv, s2 = p2 * dv;
        const double nn = n_raw > kTiny ? n_raw : kTiny;
        const double u = nu_raw / nn;
        double Tg = s2 / nn - u * u;
        if (!(Tg > 0.0)) Tg = kTiny;
        n[warp] = nn;
        nu[warp] = nu_raw;
        T[warp] = Tg;
    }
}

// ---- K2: Maxwellian + upwind implicit assembly ----------------------------
// implicit_kernels.cu:84-134.  A thread owns one cell k and kSysV velocities:
// the cell's roots and quotients are formed once instead of once per element,
// and no element index is divided.  Neighbouring threads write neighbouring k,
// so the four systems stream out coalesced.  Bound by HBM writes; 2048 x 256:
// 11.6 -> 9.7 us under ncu on one B200.
constexpr int kSysV = 8;
__global__ void __launch_bounds__(128) build_system_kernel(
    const double* __restrict__ B0, const double* __restrict__ v, const double* __restrict__ n,
    const double* __restrict__ nu, const double* __restrict__ Tg, const double* __restrict__ fl,
    const double* __restrict__ fr, int nx, int nv, double dt, double dx, double tau_tilde,
    double inv_sqrt_2pi, double* __restrict__ dl, double* __restrict__ dd,
    double* __restrict__ du, double* __restrict__ B, int jblocks) {
    const int n_inner = nx - 2;
    const int k = (int)(blockIdx.x / jblocks) * blockDim.x + threadIdx.x;
    const int j0 = (int)(blockIdx.x % jblocks) * kSysV;
    if (k >= n_inner) return;
    const int i = k + 1;
    const double ni = n[i] > kTiny ? n[i] : kTiny;
    const double Ti = Tg[i] > kTiny ? Tg[i] : kTiny;
    const double ui = nu[i] / ni;
    const double sT = sqrt(Ti);
    const double inv_tau = (ni * sT) / tau_tilde;
    const double cM = ni * inv_sqrt_2pi / sT;
    const double dti = dt * inv_tau;
    const bool ord = Ti >= 1e-200 && Ti <= 1e200;
    const double rT = ord ? recip3(Ti) : 0.0;
#pragma unroll 4
    for (int jj = 0; jj < kSysV; ++jj) {
        const int j = j0 + jj;
        if (j >= nv) break;
        const size_t t = (size_t)j * n_inner + k;
        const double vj = v[j];
        const double alpha = vj > 0.0 ? (dt / dx) * vj : 0.0;
        const double beta = vj < 0.0 ? (dt / dx) * (-vj) : 0.0;
        dd[t] = 1.0 + alpha + beta + dti;
        dl[t] = k == 0 ? 0.0 : -alpha;
        du[t] = k == n_inner - 1 ? 0.0 : -beta;
        const double diff = vj - ui;
        const double a = -0.5 * diff * diff;
        // a / Ti (-inf where u of a nearly empty cell, about 1e300, overflows a)
        double q = refined(a * rT, Ti, a, rT);
        if (!ord) q = a / Ti;
        const double fM = cM * exp(q);
        double rhs = B0[t] + dti * fM;
        if (k == 0) rhs += alpha * fl[j];
        if (k == n_inner - 1) rhs += beta * fr[j];
        B[t] = rhs;
    }
}

// ---- K5: batched 3x3 block-tridiagonal solve -------------------------------
__device__ __forceinline__ void m3mul(const double* A, const double* B, double* C) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            C[3 * i + j] = A[3 * i] * B[j] + A[3 * i + 1] * B[3 + j] + A[3 * i + 2] * B[6 + j];
}
__device__ __forceinline__ void m3vec(const double* A, const double* x, double* y) {
#pragma unroll
    for (int i = 0; i < 3; ++i) y[i] = A[3 * i] * x[0] + A[3 * i + 1] * x[1] + A[3 * i + 2] * x[2];
}
// Adjugate inverse; |det| < 1e-30 -> zero matrix
// (lo_blocktridiag/block_tridiag_kernel.cu:32-68, 248-250 convention).
__device__ __forceinline__ void m3inv(const double* M, double* Mi) {
    const double a00 = M[0], a01 = M[1], a02 = M[2], a10 = M[3], a11 = M[4], a12 = M[5],
                 a20 = M[6], a21 = M[7], a22 = M[8];
    const double c00 = (a11 * a22 - a12 * a21), c01 = -(a10 * a22 - a12 * a20),
                 c02 = (a10 * a21 - a11 * a20);
    const double c10 = -(a01 * a22 - a02 * a21), c11 = (a00 * a22 - a02 * a20),
                 c12 = -(a00 * a21 - a01 * a20);
    const double c20 = (a01 * a12 - a02 * a11), c21 = -(a00 * a12 - a02 * a10),
                 c22 = (a00 * a11 - a01 * a10);
    const double det = a00 * c00 + a01 * c01 + a02 * c02;
    if (!(fabs(det) >= 1e-30)) {
#pragma unroll
        for (int k = 0; k < 9; ++k) Mi[k] = 0.0;
        return;
    }
    const double id = 1.0 / det;
    Mi[0] = c00 * id; Mi[1] = c10 * id; Mi[2] = c20 * id;
    Mi[3] = c01 * id; Mi[4] = c11 * id; Mi[5] = c21 * id;
    Mi[6] = c02 * id; Mi[7] = c12 * id; Mi[8] = c22 * id;
}

// Partition method for batched 3x3 block-tridiagonal systems
//   A_i x_{i-1} + B_i x_i + C_i x_{i+1} = D_i,   i = 0 .. n-1 (A_0, C_{n-1} ignored).
// Rows are cut into K chunks of L rows.  Per chunk (one thread), the rows
// s..e-1 before the chunk's last row e are eliminated by block Thomas with
// the chunk's two interface unknowns xi_{k-1} = x_{s-1} and xi_k = x_e moved
// to the right-hand side, giving x_i = y_i + P_i xi_{k-1} + Q_i xi_k.  The
// chunks' last rows then form a K-row block-tridiagonal system in the xi,
// solved by parallel cyclic reduction in one CTA per system, a row per thread;
// a last pass recovers every x_i.  Singular 3x3 pivots (|det| < 1e-30)
// contribute a zero inverse, the convention of
// lo_blocktridiag/block_tridiag_kernel.cu:32-68.
//
// What bounds it: latency.  With 32-row chunks walked over global memory the
// elimination alone took 231 of 248 us for one system of 4094 rows on one B200
// (each of 62 steps waits for the row stored by the step before).  Chunks of 9
// rows in shared memory (odd, so that threads a chunk apart use different
// banks) take 16 short steps, and the longer interface system costs a step or
// two because its couplings, products of a chunk's, are small: 32 us for the
// whole call.
struct BtGeo {
    int L, K;
};
constexpr int kBtMaxK = 512;      // interface rows at most: one per thread
constexpr int kBtCta = 32;        // chunks per CTA of the elimination
constexpr int kBtSmemRow = 30;    // A (9) | B (9) | C (9) | D (3)
__host__ __device__ inline BtGeo bt_geo(int n) {
    BtGeo g;
    int L = (n + kBtMaxK - 1) / kBtMaxK;
    L = L < 9 ? 9 : L | 1;
    g.L = L;
    g.K = (n + L - 1) / L;
    return g;
}
constexpr int kBtRep = 21;  // y (3) | P (3x3) | Q (3x3) per row
// Rows that a CTA of the elimination holds at most.
__host__ __device__ inline int bt_cta_rows(int n, BtGeo g) {
    return n < kBtCta * g.L ? n : kBtCta * g.L;
}

// Block Thomas over the local rows of a chunk; the representation of row i
// replaces its D (y), A (P) and B (Q), and M^-1 C replaces C.  a, b, c, d are
// the arrays of the chunk's first row.
__device__ __forceinline__ void bt_eliminate(double* a, double* b, double* c, double* d, int nloc,
                                             bool first_chunk) {
    for (int r = 0; r < nloc; ++r) {
        double* Ai = a + 9 * r;
        double* Bi = b + 9 * r;
        double* Ci = c + 9 * r;
        double* Di = d + 3 * r;
        double M[9], ry[3], rP[9];
        for (int q = 0; q < 9; ++q) M[q] = Bi[q];
        for (int q = 0; q < 3; ++q) ry[q] = Di[q];
        if (r == 0) {
            for (int q = 0; q < 9; ++q) rP[q] = first_chunk ? 0.0 : -Ai[q];
        } else {
            double T9[9], t3[3], A9[9];
            for (int q = 0; q < 9; ++q) A9[q] = Ai[q];
            m3mul(A9, Ci - 9, T9);
            for (int q = 0; q < 9; ++q) M[q] -= T9[q];
            m3vec(A9, Di - 3, t3);
            for (int q = 0; q < 3; ++q) ry[q] -= t3[q];
            m3mul(A9, Ai - 9, T9);
            for (int q = 0; q < 9; ++q) rP[q] = -T9[q];
        }
        double Mi[9], t9[9], C9[9];
        m3inv(M, Mi);
        m3vec(Mi, ry, Di);
        m3mul(Mi, rP, t9);
        for (int q = 0; q < 9; ++q) Ai[q] = t9[q];
        for (int q = 0; q < 9; ++q) C9[q] = Ci[q];
        m3mul(Mi, C9, t9);
        for (int q = 0; q < 9; ++q) Ci[q] = t9[q];
    }
    // backward: x_i = R'_i - C'_i x_{i+1}; the last local row couples to xi_k
    for (int r = nloc - 1; r >= 0; --r) {
        double* Ai = a + 9 * r;
        double* Bi = b + 9 * r;
        const double* Ci = c + 9 * r;
        double* Di = d + 3 * r;
        if (r == nloc - 1) {
            for (int q = 0; q < 9; ++q) Bi[q] = -Ci[q];
        } else {
            double t3[3], T9[9];
            m3vec(Ci, Di + 3, t3);
            for (int q = 0; q < 3; ++q) Di[q] -= t3[q];
            m3mul(Ci, Ai + 9, T9);
            for (int q = 0; q < 9; ++q) Ai[q] -= T9[q];
            m3mul(Ci, Bi + 9, T9);
            for (int q = 0; q < 9; ++q) Bi[q] = -T9[q];
        }
    }
    // the chunk's last row is its interface unknown: y = 0, P = 0, Q = I
    for (int q = 0; q < 9; ++q) {
        a[9 * nloc + q] = 0.0;
        b[9 * nloc + q] = (q & 3) == 0 ? 1.0 : 0.0;
    }
    for (int q = 0; q < 3; ++q) d[3 * nloc + q] = 0.0;
}

// Systems that a thread solves alone, by block Thomas: those of about a chunk, for
// which the partition does the same steps in three launches, and short ones of which
// there are enough to fill the chip with a thread each.  us per call, partition and
// thread: 1024 systems of 8 rows 36 and 21, 65536 of them 393 and 59; 2048 of 16 rows
// 30 and 36, 4096 of them 44 and 36; 4096 of 32 rows 55 and 71, 8192 of them 95 and
// 75; 8192 of 64 rows 120 and 195.
inline bool bt_by_thread(int n, int batch) {
    return n <= 12 || (n <= 32 && batch >= 256 * n);
}

// A thread per system, by block Thomas.  ws: C' (9) and y (3) per row, row by row
// over all systems, so that neighbouring threads use neighbouring words.
__global__ void __launch_bounds__(64) bt_thread_kernel(const double* __restrict__ A,
                                                       const double* __restrict__ Bm,
                                                       const double* __restrict__ C,
                                                       const double* __restrict__ D, int n, int batch,
                                                       double* __restrict__ ws, double* __restrict__ X) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= batch) return;
    const size_t st = (size_t)batch;
    const double* Ai = A + (size_t)b * n * 9;
    const double* Bi = Bm + (size_t)b * n * 9;
    const double* Ci = C + (size_t)b * n * 9;
    const double* Di = D + (size_t)b * n * 3;
    double* Xi = X + (size_t)b * n * 3;
    double* w = ws + b;
    double cp[9], y[3];
#pragma unroll
    for (int q = 0; q < 9; ++q) cp[q] = 0.0;
    y[0] = y[1] = y[2] = 0.0;
    for (int r = 0; r < n; ++r) {
        double M[9], t9[9], t3[3], ry[3], Mi[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) M[q] = Bi[9 * r + q];
#pragma unroll
        for (int q = 0; q < 3; ++q) ry[q] = Di[3 * r + q];
        if (r > 0) {
            double a[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) a[q] = Ai[9 * r + q];
            m3mul(a, cp, t9);
#pragma unroll
            for (int q = 0; q < 9; ++q) M[q] -= t9[q];
            m3vec(a, y, t3);
#pragma unroll
            for (int q = 0; q < 3; ++q) ry[q] -= t3[q];
        }
        m3inv(M, Mi);
        m3vec(Mi, ry, y);
        if (r + 1 < n) {
            double c[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) c[q] = Ci[9 * r + q];
            m3mul(Mi, c, cp);
#pragma unroll
            for (int q = 0; q < 9; ++q) w[(12 * (size_t)r + q) * st] = cp[q];
#pragma unroll
            for (int q = 0; q < 3; ++q) w[(12 * (size_t)r + 9 + q) * st] = y[q];
        }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) Xi[3 * (n - 1) + q] = y[q];
    for (int r = n - 2; r >= 0; --r) {
        double t3[3];
#pragma unroll
        for (int q = 0; q < 9; ++q) cp[q] = w[(12 * (size_t)r + q) * st];
        m3vec(cp, y, t3);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            y[q] = w[(12 * (size_t)r + 9 + q) * st] - t3[q];
            Xi[3 * r + q] = y[q];
        }
    }
}

// A CTA of one warp and kBtCta chunks (grid: chunk groups x systems).  rep, per
// system: y (3 n) | P (9 n) | Q (9 n); cpw: 9 n of scratch.  With kSmem the
// rows are staged through shared memory by coalesced copies, otherwise worked
// on in rep and cpw.
template <bool kSmem>
__global__ void __launch_bounds__(kBtCta) bt_local_kernel(const double* __restrict__ A,
                                                          const double* __restrict__ Bm,
                                                          const double* __restrict__ C,
                                                          const double* __restrict__ D, int n,
                                                          double* __restrict__ rep,
                                                          double* __restrict__ cpw) {
    extern __shared__ __align__(16) double bt_sm[];
    const BtGeo G = bt_geo(n);
    const int groups = (G.K + kBtCta - 1) / kBtCta;
    const int b = (int)(blockIdx.x / groups), g = (int)(blockIdx.x % groups);
    const int lane = threadIdx.x;
    const int r0 = g * kBtCta * G.L;                              // rows of the CTA
    const int nr = n - r0 < kBtCta * G.L ? n - r0 : kBtCta * G.L;
    const size_t mo = ((size_t)b * n + r0) * 9, vo = ((size_t)b * n + r0) * 3;
    double* gy = rep + (size_t)b * n * kBtRep + 3 * (size_t)r0;
    double* gP = rep + (size_t)b * n * kBtRep + 3 * (size_t)n + 9 * (size_t)r0;
    double* gQ = gP + 9 * (size_t)n;
    double* gC = cpw + (size_t)b * n * 9 + 9 * (size_t)r0;
    const int rows = bt_cta_rows(n, G);
    double* a = kSmem ? bt_sm : gP;
    double* bb = kSmem ? bt_sm + 9 * (size_t)rows : gQ;
    double* c = kSmem ? bt_sm + 18 * (size_t)rows : gC;
    double* d = kSmem ? bt_sm + 27 * (size_t)rows : gy;
    if (kSmem) {
        for (int q = lane; q < 9 * nr; q += kBtCta) {
            cp_async8(a + q, A + mo + q);
            cp_async8(bb + q, Bm + mo + q);
            cp_async8(c + q, C + mo + q);
        }
        for (int q = lane; q < 3 * nr; q += kBtCta) cp_async8(d + q, D + vo + q);
        cp_async_commit();
        cp_async_wait_all();
    } else {
        for (int q = lane; q < 9 * nr; q += kBtCta) {
            a[q] = A[mo + q];
            bb[q] = Bm[mo + q];
            c[q] = C[mo + q];
        }
        for (int q = lane; q < 3 * nr; q += kBtCta) d[q] = D[vo + q];
    }
    __syncthreads();
    const int s = lane * G.L;  // within the CTA's rows
    if (s < nr) {
        const int e = (s + G.L < nr ? s + G.L : nr) - 1;
        bt_eliminate(a + 9 * s, bb + 9 * s, c + 9 * s, d + 3 * s, e - s, r0 + s == 0);
    }
    if (kSmem) {
        __syncthreads();
        for (int q = lane; q < 9 * nr; q += kBtCta) {
            gP[q] = a[q];
            gQ[q] = bb[q];
        }
        for (int q = lane; q < 3 * nr; q += kBtCta) gy[q] = d[q];
    }
}

// Interface system of one system per CTA, a row per thread in registers; one
// exchange buffer: al (9) | be^-1 (9) | ga (9) | de (3) per row.
__global__ void __launch_bounds__(kBtMaxK) bt_reduced_kernel(const double* __restrict__ A,
                                                             const double* __restrict__ Bm,
                                                             const double* __restrict__ C,
                                                             const double* __restrict__ D, int n,
                                                             const double* __restrict__ rep,
                                                             double* __restrict__ xi) {
    extern __shared__ __align__(16) double bt_sm[];
    const BtGeo G = bt_geo(n);
    const int b = blockIdx.x, K = G.K, k = threadIdx.x, T = blockDim.x;
    const bool on = k < K;
    const size_t mo = (size_t)b * n * 9, vo = (size_t)b * n * 3;
    const double* gy = rep + (size_t)b * n * kBtRep;
    const double* gP = gy + 3 * (size_t)n;
    const double* gQ = gP + 9 * (size_t)n;
    double al[9], be[9], ga[9], de[3];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        al[q] = ga[q] = 0.0;
        be[q] = (q & 3) == 0 ? 1.0 : 0.0;
    }
    de[0] = de[1] = de[2] = 0.0;
    if (on) {
        const int s = k * G.L;
        const int e = (s + G.L < n ? s + G.L : n) - 1;
        double T9[9], t3[3], M9[9], V[9], v3[3];
#pragma unroll
        for (int q = 0; q < 9; ++q) be[q] = Bm[mo + 9 * (size_t)e + q];
#pragma unroll
        for (int q = 0; q < 3; ++q) de[q] = D[vo + 3 * (size_t)e + q];
        if (e > 0) {
#pragma unroll
            for (int q = 0; q < 9; ++q) M9[q] = A[mo + 9 * (size_t)e + q];
            if (e > s) {  // x_{e-1} = y + P xi_{k-1} + Q xi_k
#pragma unroll
                for (int q = 0; q < 9; ++q) V[q] = gP[9 * (size_t)(e - 1) + q];
                m3mul(M9, V, al);
#pragma unroll
                for (int q = 0; q < 9; ++q) V[q] = gQ[9 * (size_t)(e - 1) + q];
                m3mul(M9, V, T9);
#pragma unroll
                for (int q = 0; q < 9; ++q) be[q] += T9[q];
#pragma unroll
                for (int q = 0; q < 3; ++q) v3[q] = gy[3 * (size_t)(e - 1) + q];
                m3vec(M9, v3, t3);
#pragma unroll
                for (int q = 0; q < 3; ++q) de[q] -= t3[q];
            } else {
#pragma unroll
                for (int q = 0; q < 9; ++q) al[q] = M9[q];
            }
        }
        if (k + 1 < K) {  // x_{e+1} = y + P xi_k + Q xi_{k+1}
#pragma unroll
            for (int q = 0; q < 9; ++q) M9[q] = C[mo + 9 * (size_t)e + q];
#pragma unroll
            for (int q = 0; q < 9; ++q) V[q] = gP[9 * (size_t)(e + 1) + q];
            m3mul(M9, V, T9);
#pragma unroll
            for (int q = 0; q < 9; ++q) be[q] += T9[q];
#pragma unroll
            for (int q = 0; q < 9; ++q) V[q] = gQ[9 * (size_t)(e + 1) + q];
            m3mul(M9, V, ga);
#pragma unroll
            for (int q = 0; q < 3; ++q) v3[q] = gy[3 * (size_t)(e + 1) + q];
            m3vec(M9, v3, t3);
#pragma unroll
            for (int q = 0; q < 3; ++q) de[q] -= t3[q];
        }
    }
    double bi[9];
    for (int st = 1; st < K; st <<= 1) {
        m3inv(be, bi);
        double nb = 0.0, nc = 0.0;
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            nb += fabs(bi[q]);
            nc += fabs(al[q]) + fabs(ga[q]);
        }
        // (a singular block, whose inverse is zero, is not decoupled yet)
        const bool dec = nb * nc <= 8.673617379884035e-19 && (nb > 0.0 || nc == 0.0);  // 2^-60
        if (__syncthreads_and(dec)) {  // (also: the reads of the step before are done)
            // Every row is decoupled to below double rounding of the largest value.
            // Where a solution decays, a value may be far below that and consist of
            // what the coupling brings: done if, entry by entry, the coupling to the
            // neighbours' values is small against the row's own (the Jacobi iteration
            // scaled by them contracts by 2^-58), or vanishes in a double's range.
            // Going on to the latter always took four more steps, 31 -> 39 us for one
            // system of 4094 rows; the comparison takes none.
            double xh[3];
            m3vec(bi, de, xh);
#pragma unroll
            for (int q = 0; q < 3; ++q) bt_sm[q * T + k] = fabs(xh[q]);
            __syncthreads();
            double g[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                g[i] = 0.0;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    if (k >= st) g[i] = fma(fabs(al[3 * i + q]), bt_sm[q * T + k - st], g[i]);
                    if (k + st < K) g[i] = fma(fabs(ga[3 * i + q]), bt_sm[q * T + k + st], g[i]);
                }
            }
            bool own = true;
#pragma unroll
            for (int i = 0; i < 3; ++i)
                own &= fabs(bi[3 * i]) * g[0] + fabs(bi[3 * i + 1]) * g[1] + fabs(bi[3 * i + 2]) * g[2] <=
                       3.469446951953614e-18 * fabs(xh[i]);
            // (a value that is not finite goes on: it has to reach every row)
            own |= nb * nc <= 1e-270 && isfinite(xh[0]) && isfinite(xh[1]) && isfinite(xh[2]);
            if (__syncthreads_and(own || !on)) break;
        }
        // (element-major: neighbouring threads use neighbouring words)
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            bt_sm[q * T + k] = al[q];
            bt_sm[(9 + q) * T + k] = bi[q];
            bt_sm[(18 + q) * T + k] = ga[q];
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) bt_sm[(27 + q) * T + k] = de[q];
        __syncthreads();
        double e1[9], V[9], T9[9], v3[3], t3[3], na[9];
        const bool lo = k >= st && on, hi = k + st < K;
        const int kl = lo ? k - st : k, kh = hi ? k + st : k;
#pragma unroll
        for (int q = 0; q < 9; ++q) V[q] = lo ? bt_sm[(9 + q) * T + kl] : 0.0;
        m3mul(al, V, e1);
#pragma unroll
        for (int q = 0; q < 9; ++q) V[q] = bt_sm[q * T + kl];
        m3mul(e1, V, T9);
#pragma unroll
        for (int q = 0; q < 9; ++q) na[q] = -T9[q];
#pragma unroll
        for (int q = 0; q < 9; ++q) V[q] = bt_sm[(18 + q) * T + kl];
        m3mul(e1, V, T9);
#pragma unroll
        for (int q = 0; q < 9; ++q) be[q] -= T9[q];
#pragma unroll
        for (int q = 0; q < 3; ++q) v3[q] = bt_sm[(27 + q) * T + kl];
        m3vec(e1, v3, t3);
#pragma unroll
        for (int q = 0; q < 3; ++q) de[q] -= t3[q];
#pragma unroll
        for (int q = 0; q < 9; ++q) V[q] = hi ? bt_sm[(9 + q) * T + kh] : 0.0;
        m3mul(ga, V, e1);
#pragma unroll
        for (int q = 0; q < 9; ++q) V[q] = bt_sm[(18 + q) * T + kh];
        m3mul(e1, V, T9);
#pragma unroll
        for (int q = 0; q < 9; ++q) ga[q] = -T9[q];
#pragma unroll
        for (int q = 0; q < 9; ++q) V[q] = bt_sm[q * T + kh];
        m3mul(e1, V, T9);
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            be[q] -= T9[q];
            al[q] = na[q];
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) v3[q] = bt_sm[(27 + q) * T + kh];
        m3vec(e1, v3, t3);
#pragma unroll
        for (int q = 0; q < 3; ++q) de[q] -= t3[q];
    }
    if (on) {
        m3inv(be, bi);
        double x[3];
        m3vec(bi, de, x);
#pragma unroll
        for (int q = 0; q < 3; ++q) xi[((size_t)b * K + k) * 3 + q] = x[q];
    }
}

// One thread per unknown: x = y + P xi_{k-1} + Q xi_k.
__global__ void __launch_bounds__(128) bt_recover_kernel(int n, int batch,
                                                         const double* __restrict__ rep,
                                                         const double* __restrict__ xi,
                                                         double* __restrict__ X) {
    const BtGeo G = bt_geo(n);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)batch * n * 3) return;
    const int b = (int)(t / (3 * (long long)n));
    const int u = (int)(t - 3 * (long long)n * b), i = u / 3, c = u - 3 * i;
    const int k = i / G.L;
    const double* gy = rep + (size_t)b * n * kBtRep;
    const double* P = gy + 3 * (size_t)n + 9 * (size_t)i + 3 * c;
    const double* Q = P + 9 * (size_t)n;
    const double* xl = xi + ((size_t)b * G.K + (k > 0 ? k - 1 : 0)) * 3;
    const double* xr = xi + ((size_t)b * G.K + k) * 3;
    const double a = P[0] * xl[0] + P[1] * xl[1] + P[2] * xl[2];
    const double e = Q[0] * xr[0] + Q[1] * xr[1] + Q[2] * xr[2];
    X[t] = gy[u] + (k > 0 ? a : 0.0) + e;
}

// ---- Maxwellian of per-row moments -----------------------------------------
// bgk1d_utils/general/bgk1d_maxwellian.py:7-33, element for element:
// coeff = n/sqrt(2 pi T) (n * inv_sqrt_2pi / sqrt(T)), e = (v-u)^2 * (-0.5/T),
// f = exp(e) * coeff.  One thread per (i, j), j fastest (coalesced rows).
__global__ void __launch_bounds__(256) maxwellian_kernel(const double* __restrict__ n,
                                                         const double* __restrict__ u,
                                                         const double* __restrict__ T,
                                                         const double* __restrict__ v, int nx,
                                                         int nv, double* __restrict__ f) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nx * nv) return;
    const int i = (int)(t / nv), j = (int)(t % nv);
    const double Ti = T[i];
    const double coeff = (n[i] * kInvSqrt2Pi) / sqrt(Ti);
    const double invT = 0.5 / Ti;
    const double d = v[j] - u[i];
    f[t] = exp((d * d) * (-invT)) * coeff;
}

// ---- raw velocity moments (no clamps) ---------------------------------------
// Row densities of mass, momentum and energy: (sum f dv, sum f v dv,
// sum f v^2/2 dv), one warp per row, fixed butterfly order.  Used for the
// conservation totals of a state and as calculate_moments' raw sums
// (bgk1d_utils/general/bgk1d_compute_moments.py:7-17).
__global__ void __launch_bounds__(256) row_moments_kernel(const double* __restrict__ f,
                                                          const double* __restrict__ v, int nx,
                                                          int nv, double dv,
                                                          double* __restrict__ out) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= nx) return;
    const double* row = f + (size_t)warp * nv;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    for (int j = lane; j < nv; j += 32) {
        const double x = row[j], vj = v[j];
        p0 += x;
        p1 += x * vj;
        p2 += x * (vj * vj);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        p0 += __shfl_xor_sync(0xffffffffu, p0, o);
        p1 += __shfl_xor_sync(0xffffffffu, p1, o);
        p2 += __shfl_xor_sync(0xffffffffu, p2, o);
    }
    if (lane == 0) {
        out[3 * (size_t)warp + 0] = p0 * dv;
        out[3 * (size_t)warp + 1] = p1 * dv;
        out[3 * (size_t)warp + 2] = 0.5 * (p2 * dv);
    }
}

// Evaluates the device math helpers on an array (numerical self-test).
__global__ void math_selftest_kernel(int kind, const double* __restrict__ x, double* __restrict__ y,
                                     int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double root, inv;
    switch (kind) {
        case 0: y[i] = exp_nonpos(x[i]); break;
        case 1: y[i] = recip_ge1(x[i]); break;
        case 2: y[i] = rows::exp_neg(x[i]); break;
        case 3: y[i] = recip3(x[i]); break;
        case 4: y[i] = div_nr(x[i], y[i]); break;
        default:
            sqrt_nr(x[i], root, inv);
            y[i] = kind == 5 ? root : inv;
    }
}

}  // namespace keq

namespace {
keq_status launch_status() {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        keq_internal_set_cuda_error(e);
        return KEQ_ERR_CUDA;
    }
    return KEQ_OK;
}
}  // namespace

extern "C" {

keq_status keq_moments_n_nu_T(const double* f, const double* v, int32_t nx, int32_t nv, double dv,
                              double* n, double* nu, double* T, keq_stream_t stream) {
    if (!f || !v || !n || !nu || !T || nx < 1 || nv < 1) return KEQ_ERR_INVALID;
    const long long threads = (long long)nx * 32;
    const int blocks = (int)((threads + 255) / 256);
    keq::moments_kernel<<<blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(f, v, nx, nv,
                                                                                   dv, n, nu, T);
    return launch_status();
}

keq_status keq_build_system_from_moments(const double* B0, const double* v, int32_t nx,
                                         int32_t nv, double dt, double dx, double tau_tilde,
                                         double inv_sqrt_2pi, const double* n, const double* nu,
                                         const double* T, const double* f_bc_l,
                                         const double* f_bc_r, double* dl, double* dd,
                                         double* du, double* B, keq_stream_t stream) {
    if (!B0 || !v || !n || !nu || !T || !f_bc_l || !f_bc_r || !dl || !dd || !du || !B)
        return KEQ_ERR_INVALID;
    if (nx < 3 || nv < 1) return KEQ_ERR_INVALID;
    const long long jblocks = (nv + keq::kSysV - 1) / keq::kSysV;
    const long long blocks = ((long long)(nx - 2) + 127) / 128 * jblocks;
    if (blocks > 0x7fffffffll) return KEQ_ERR_INVALID;
    keq::build_system_kernel<<<(unsigned)blocks, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        B0, v, n, nu, T, f_bc_l, f_bc_r, nx, nv, dt, dx, tau_tilde, inv_sqrt_2pi, dl, dd, du, B,
        (int)jblocks);
    return launch_status();
}

keq_status keq_maxwellian(const double* n, const double* u, const double* T, const double* v,
                          int32_t nx, int32_t nv, double* f, keq_stream_t stream) {
    if (!n || !u || !T || !v || !f || nx < 1 || nv < 1) return KEQ_ERR_INVALID;
    const long long total = (long long)nx * nv;
    keq::maxwellian_kernel<<<(unsigned)((total + 255) / 256), 256, 0,
                             reinterpret_cast<cudaStream_t>(stream)>>>(n, u, T, v, nx, nv, f);
    return launch_status();
}

keq_status keq_row_moments(const double* f, const double* v, int32_t nx, int32_t nv, double dv,
                           double* out, keq_stream_t stream) {
    if (!f || !v || !out || nx < 1 || nv < 1) return KEQ_ERR_INVALID;
    const long long threads = (long long)nx * 32;
    keq::row_moments_kernel<<<(unsigned)((threads + 255) / 256), 256, 0,
                              reinterpret_cast<cudaStream_t>(stream)>>>(f, v, nx, nv, dv, out);
    return launch_status();
}

keq_status keq_math_selftest(int32_t kind, const double* x, double* y, int32_t n,
                             keq_stream_t stream) {
    if (!x || !y || n < 0 || kind < 0 || kind > 6) return KEQ_ERR_INVALID;
    if (n == 0) return KEQ_OK;
    keq::math_selftest_kernel<<<(n + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        kind, x, y, n);
    return launch_status();
}

keq_status keq_gtsv_workspace_size(int32_t n, int32_t batch, size_t* bytes) {
    if (!bytes || n < 0 || batch < 0) return KEQ_ERR_INVALID;
    *bytes = sizeof(double) * (size_t)(n > 0 ? n : 1) * (size_t)(batch > 0 ? batch : 1);
    return KEQ_OK;
}

keq_status keq_gtsv_strided_inplace(const double* dl, const double* d, const double* du,
                                    double* B, int32_t n, int32_t batch, void* workspace,
                                    size_t workspace_bytes, keq_stream_t stream) {
    if (n < 0 || batch < 0) return KEQ_ERR_INVALID;
    if (n == 0 || batch == 0) return KEQ_OK;
    if (!dl || !d || !du || !B || !workspace) return KEQ_ERR_INVALID;
    size_t need = 0;
    keq_gtsv_workspace_size(n, batch, &need);
    if (workspace_bytes < need || reinterpret_cast<uintptr_t>(workspace) % 8)
        return KEQ_ERR_WORKSPACE;
    const cudaError_t e = keq::launch_gtsv(dl, d, du, B, n, batch, static_cast<double*>(workspace),
                                           reinterpret_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) {
        keq_internal_set_cuda_error(e);
        return KEQ_ERR_CUDA;
    }
    return KEQ_OK;
}

keq_status keq_block_tridiag_workspace_size(int32_t n, int32_t batch, size_t* bytes) {
    if (!bytes || n < 0 || batch < 0) return KEQ_ERR_INVALID;
    const size_t nn = (size_t)(n > 0 ? n : 1), bb = (size_t)(batch > 0 ? batch : 1);
    const keq::BtGeo G = keq::bt_geo(n > 0 ? n : 1);
    *bytes = sizeof(double) * (nn * bb * (keq::kBtRep + 9) + (size_t)G.K * bb * 3) + 256;
    return KEQ_OK;
}

keq_status keq_block_tridiag_solve(const double* A, const double* B, const double* C,
                                   const double* D, double* X, int32_t n, int32_t batch,
                                   void* workspace, size_t workspace_bytes,
                                   keq_stream_t stream) {
    if (n < 0 || batch < 0) return KEQ_ERR_INVALID;
    if (n == 0 || batch == 0) return KEQ_OK;
    if (!A || !B || !C || !D || !X || !workspace) return KEQ_ERR_INVALID;
    size_t need = 0;
    keq_block_tridiag_workspace_size(n, batch, &need);
    if (workspace_bytes < need || reinterpret_cast<uintptr_t>(workspace) % 8)
        return KEQ_ERR_WORKSPACE;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const keq::BtGeo G = keq::bt_geo(n);
    double* rep = static_cast<double*>(workspace);
    double* cpw = rep + (size_t)n * batch * keq::kBtRep;
    double* xi = cpw + (size_t)n * batch * 9;
    if (keq::bt_by_thread(n, batch)) {
        keq::bt_thread_kernel<<<(unsigned)(((long long)batch + 63) / 64), 64, 0, s>>>(A, B, C, D, n, batch, rep, X);
        return launch_status();
    }
    const long long groups = (long long)batch * ((G.K + keq::kBtCta - 1) / keq::kBtCta);
    const size_t local = sizeof(double) * keq::kBtSmemRow * (size_t)keq::bt_cta_rows(n, G);
    if (local <= 224 * 1024) {
        cudaFuncSetAttribute(keq::bt_local_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             224 * 1024);
        keq::bt_local_kernel<true><<<(unsigned)groups, keq::kBtCta, local, s>>>(A, B, C, D, n, rep, cpw);
    } else {
        keq::bt_local_kernel<false><<<(unsigned)groups, keq::kBtCta, 0, s>>>(A, B, C, D, n, rep, cpw);
    }
    const int T = (G.K + 31) / 32 * 32;
    const size_t smem = sizeof(double) * keq::kBtSmemRow * (size_t)T;
    cudaFuncSetAttribute(keq::bt_reduced_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(double) * keq::kBtSmemRow * keq::kBtMaxK));
    keq::bt_reduced_kernel<<<batch, T, smem, s>>>(A, B, C, D, n, rep, xi);
    const long long nrow = (long long)batch * n * 3;
    keq::bt_recover_kernel<<<(unsigned)((nrow + 127) / 128), 128, 0, s>>>(n, batch, rep, xi, X);
    return launch_status();
}

}  // extern "C"
