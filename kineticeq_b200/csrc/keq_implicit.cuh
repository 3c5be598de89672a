// keq_implicit.cuh -- what the implicit step kernels share: the instance
// and plan records on the device, the moment and coefficient formulas, the
// Anderson coefficient solve and the phase trace.
//   keq_implicit.cu       tiles with a decoupled look-back (any v_max dt/dx and
//                         the mixed-precision form); plan construction
//   keq_implicit_rows.cu  row blocks owned by one CTA (bounded v_max dt/dx)
//   keq_implicit_solo.cu  the same for one instance with all blocks resident
#pragma once

#include <math.h>

#include "keq_common.cuh"
#include "keq_internal.h"
#include "keq_tile.cuh"

namespace keq {

constexpr int kMaxAACols = 8;            // Anderson ring columns (aa_m <= 7)
constexpr int kMaxima = 5;               // PlanDev::maxima
constexpr int kMaxPairs = kMaxAACols * (kMaxAACols + 1) / 2;

struct ImpInst {
    int nx, nv, n_inner, kp;
    int nt_neg, nvt, nchunks, nrb;
    int rows, pad0;  // rows per tile (R)
    long long tile_off, rb_off;
    double dx, dv, dt, tau_tilde, dtdx, u_max;
    int picard_iter, conv_type, fixed_iters, pad1;
    double tol, abs_tol;
    int aa_on, aa_cols, aa_stride, aa_start;
    double aa_beta, aa_reg, aa_alpha_max;
    int mixed, pad2;  // mixed-precision form: FP32 sweeps, then FP64 sweeps
    double tol32;     // Picard tolerance that ends the FP32 sweeps
    const double* v;
    const double* f_in;
    double* f_out;
    keq_step_stats* stats;
    const int* enable;  // optional device flag: 0 = leave this instance untouched this step
    // workspace carve
    double* W;       // 3*nx  : n | nu | T   (W^(m))
    double* Wn;      // 3*nx  : moments of the newest iterate (unfloored)
    double* Wc;      // 4*nx  : per-row (u, -1/(2T), n/sqrt(2 pi T), dt/tau)
    double* Wb;      // 8     : moments of the two boundary rows
    double* part;    // nvt*n_inner*kPartQ
    double* agg;     // ntiles*64 : tile maps (P | Y per lane)
    double* inc;     // ntiles*32 : tile inclusive values (carry out)
    unsigned long long* flag;  // ntiles : (epoch << 2) | {agg, inc}
    unsigned* rbcnt; // picard_iter*nrb  : rows x v-tiles of a row block done
    double* res;     // 2*picard_iter : std / rel residual slots
    int* st;         // picard_iter   : 1 if active in iteration m
    int* nonfin;     // picard_iter   : non-finite flag of iterate m+1
    double* aaG;     // aa_cols * 3*n_inner
    double* aaR;     // aa_cols * 3*n_inner
    double* gpart;   // 2 * kMaxPairs * nrb : Gram partials of the row blocks, pair-major
    double* alpha;   // picard_iter * kMaxAACols
    unsigned* rbdone;// picard_iter
    float* fn32;     // nx*nv (mixed form): f^n in FP32, written by P1
    float* x32;      // nx*nv (mixed form): the FP32 iterate, updated in place
    // row-block kernels (keq_rows.cuh)
    int rblk, nblk;  // rows per block, blocks
    int kmax, pad3;  // blocks a carry is folded over at most
    long long item_off;
    double2* xch;    // 2*nblk*nvt*32 : block maps (P, Y) per lane, by iteration parity
                     // (solo kernel: one set of tagged maps, the same size)
    double* xin;     // nblk*nvt*32 : inflow of each block's tiles in the last iteration
    unsigned* nanspan;  // 2*(picard_iter+1): of iteration m's W, blk+1 of the last and nblk-blk of
                        // the first block with NaN rows
    double* scal;    // picard_iter+3 : max |f^n|, max Maxwellian coefficient of W^(0), max n by iteration
};

// Device header of an implicit plan (starts with the common PlanHead).
struct PlanDev {
    PlanHead head;
    int n_inst;
    int max_iter;
    long long total_tiles;
    long long total_rb;
    ImpInst* inst;
    long long* tile_off;  // n_inst+1
    long long* rb_off;    // n_inst+1
    unsigned* tickets;    // max_iter : tile (item) claims of iteration m
    // row-block kernel: an item is one row block of one instance
    long long total_items;
    long long* item_off;  // n_inst+1
    int nslot;            // partial-sum slots per CTA
    int buf_rows;         // rows of a tile buffer: the most that a block has
    // solo kernel (keq_implicit_solo.cu)
    ulonglong2* maps;     // nblk * nvt * 64 : second set of block maps, tagged words (the first is in xch)
    unsigned long long arrivals;  // launch_barrier
    // by launch parity: max |f^n|, max Maxwellian coefficient, max n of W^(0); blk + 1
    // of the last and nblk - blk of the first block with NaN rows
    double maxima[2][kMaxima];
    ulonglong2* gather;   // 2 * nblk * 4 : per block residuals and bounds, tagged words
    ulonglong2* gram;     // 2 * kMaxPairs * nblk : Gram partials, tagged words
};

__device__ __forceinline__ bool inst_enabled(const ImpInst& I) {
    return I.enable == nullptr || __ldcg(I.enable) != 0;
}

// Anderson call z (after Picard iteration z) applies the combination iff
// z+1 >= start, (z+1-start) % stride == 0 and its history length
// min(z+1, cols) >= 2 (bgk1d_implicit_cuda_kernel.py:247-282, bgk1d_aa_cpu.py:131).
__device__ __forceinline__ bool aa_applies(const ImpInst& I, int z) {
    const int mh = (z + 1) < I.aa_cols ? (z + 1) : I.aa_cols;
    return I.aa_on && (z + 1) >= I.aa_start && ((z + 1 - I.aa_start) % I.aa_stride == 0) &&
           mh >= 2;
}

// Per-row solve coefficients from (n, nu, T): implicit_kernels.cu:115-125
// (n, T clamped at 1e-300; 1/tau = n sqrt(T)/tau_tilde).
__device__ __forceinline__ void row_coeffs(double tau_tilde, double dt, double n, double nu,
                                           double T, double* c4) {
    const double ni = n > kTiny ? n : kTiny;
    const double Ti = T > kTiny ? T : kTiny;
    const double ui = nu / ni;
    const double sT = sqrt(Ti);
    const double inv_tau = (ni * sT) / tau_tilde;
    c4[0] = ui;
    c4[1] = -0.5 / Ti;
    c4[2] = ni * kInvSqrt2Pi / sT;
    c4[3] = dt * inv_tau;
}

// C1/K1 moment semantics from raw sums.
__device__ __forceinline__ void moments_from_sums(double s0, double s1, double s2, double dv,
                                                  double* n, double* nu, double* T) {
    const double n_raw = s0 * dv;
    const double nu_raw = s1 * dv;
    const double s2d = s2 * dv;
    const double nv_ = n_raw > kTiny ? n_raw : kTiny;
    const double u = nu_raw / nv_;
    double Tg = s2d / nv_ - u * u;
    if (!(Tg > 0.0)) Tg = kTiny;
    *n = nv_;
    *nu = nu_raw;
    *T = Tg;
}

__device__ __forceinline__ double clamp_min_t(double x, double lo) {
    return (x != x || x >= lo) ? x : lo;
}

// Solve coefficients of a row from (n, nu, T) with the short division and root
// (div_nr, sqrt_nr).
__device__ __forceinline__ void row_coeffs_nr(double tau_tilde, double dt, double n, double nu,
                                              double T, double* c4) {
    const double ni = n > kTiny ? n : kTiny;
    const double Ti = T > kTiny ? T : kTiny;
    double sT, y;
    sqrt_nr(Ti, sT, y);
    const double a = ni * kInvSqrt2Pi;
    c4[0] = div_nr(nu, ni);
    c4[1] = -div_nr(0.5, Ti);
    c4[2] = refined(a * y, sT, a, y);
    c4[3] = dt * div_nr(ni * sT, tau_tilde);
}

// Moments (n, nu, T) of raw sums and the coefficients of the moments floored
// at `fl` (n and T).  In the ordinary range one straight line of code: the two
// reciprocals and the root are shared and independent steps overlap, which
// matters because a single warp runs this with every CTA waiting for it.
__device__ __forceinline__ void moments_and_coeffs(double s0, double s1, double s2, double dv,
                                                   double dt, double tau_tilde, double fl, double* w3,
                                                   double* c4) {
    const double n = s0 * dv, nu = s1 * dv, e2 = s2 * dv;
    const double rn = recip3(n), rt = recip3(tau_tilde);
    double u = nu * rn, e = e2 * rn;
    u = fma(fma(-u, n, nu), rn, u);
    e = fma(fma(-e, n, e2), rn, e);
    const double T = e - u * u;
    if (n >= 1e-12 && n <= 1e100 && T >= 1e-12 && T <= 1e100 && tau_tilde >= 1e-100 &&
        tau_tilde <= 1e100) {  // floors (at most 1e-12) do not act
        w3[0] = n;
        w3[1] = nu;
        w3[2] = T;
        double y;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(T));
        const double g = fma(-T * y, y, 1.0);
        y = fma(y * g, fma(g, 0.375, 0.5), y);
        double sT = T * y;
        sT = fma(fma(-sT, sT, T), 0.5 * y, sT);
        const double a = n * kInvSqrt2Pi, q = a * y, p = n * sT;
        const double it0 = p * rt;
        const double h0 = 0.5 * y * y;
        c4[0] = u;
        c4[1] = -fma(fma(-h0, T, 0.5), y * y, h0);
        c4[2] = fma(fma(-q, sT, a), y, q);
        c4[3] = dt * fma(fma(-it0, tau_tilde, p), rt, it0);
        return;
    }
    moments_from_sums(s0, s1, s2, dv, &w3[0], &w3[1], &w3[2]);
    row_coeffs(tau_tilde, dt, clamp_min_t(w3[0], fl), w3[1], clamp_min_t(w3[2], fl), c4);
}

// ---- Anderson: small symmetric solve (Cholesky, min-norm fall-back) -------
// torch.linalg.cholesky / cholesky_solve with the lstsq fall-back of
// bgk1d_aa_cpu.py:93-97; the fall-back here is a Jacobi eigen pseudo-inverse.
static __device__ __noinline__ void aa_small_solve(int m, double* A, double* x) {
    double L[kMaxAACols * kMaxAACols];
    double yv[kMaxAACols];
    bool ok = true;
    for (int i = 0; i < kMaxAACols * kMaxAACols; ++i) L[i] = 0.0;
    for (int j = 0; j < m && ok; ++j) {
        double s = A[j * m + j];
        for (int k = 0; k < j; ++k) s -= L[j * m + k] * L[j * m + k];
        if (!(s > 0.0)) { ok = false; break; }
        const double ljj = sqrt(s);
        L[j * m + j] = ljj;
        for (int i = j + 1; i < m; ++i) {
            double t = A[i * m + j];
            for (int k = 0; k < j; ++k) t -= L[i * m + k] * L[j * m + k];
            L[i * m + j] = t / ljj;
        }
    }
    if (ok) {
        for (int i = 0; i < m; ++i) {
            double t = 1.0;
            for (int k = 0; k < i; ++k) t -= L[i * m + k] * yv[k];
            yv[i] = t / L[i * m + i];
        }
        for (int i = m - 1; i >= 0; --i) {
            double t = yv[i];
            for (int k = i + 1; k < m; ++k) t -= L[k * m + i] * x[k];
            x[i] = t / L[i * m + i];
        }
        return;
    }
    double a[kMaxAACols * kMaxAACols], V[kMaxAACols * kMaxAACols];
    for (int i = 0; i < m * m; ++i) a[i] = A[i];
    for (int i = 0; i < m; ++i)
        for (int j = 0; j < m; ++j) V[i * m + j] = (i == j) ? 1.0 : 0.0;
    for (int sweep = 0; sweep < 64; ++sweep) {
        double off = 0.0;
        for (int p = 0; p < m; ++p)
            for (int q = p + 1; q < m; ++q) off += a[p * m + q] * a[p * m + q];
        if (!(off > 1e-300)) break;
        for (int p = 0; p < m; ++p)
            for (int q = p + 1; q < m; ++q) {
                const double apq = a[p * m + q];
                if (apq == 0.0) continue;
                const double th = (a[q * m + q] - a[p * m + p]) / (2.0 * apq);
                const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
                const double cs = 1.0 / sqrt(t * t + 1.0), sn = t * cs;
                for (int k = 0; k < m; ++k) {
                    const double akp = a[k * m + p], akq = a[k * m + q];
                    a[k * m + p] = cs * akp - sn * akq;
                    a[k * m + q] = sn * akp + cs * akq;
                }
                for (int k = 0; k < m; ++k) {
                    const double apk = a[p * m + k], aqk = a[q * m + k];
                    a[p * m + k] = cs * apk - sn * aqk;
                    a[q * m + k] = sn * apk + cs * aqk;
                }
                for (int k = 0; k < m; ++k) {
                    const double vkp = V[k * m + p], vkq = V[k * m + q];
                    V[k * m + p] = cs * vkp - sn * vkq;
                    V[k * m + q] = sn * vkp + cs * vkq;
                }
            }
    }
    double lmax = 0.0;
    for (int i = 0; i < m; ++i) lmax = fmax(lmax, fabs(a[i * m + i]));
    const double cut = lmax * (double)m * 2.220446049250313e-16;
    for (int i = 0; i < m; ++i) x[i] = 0.0;
    for (int k = 0; k < m; ++k) {
        const double lam = a[k * m + k];
        if (!(fabs(lam) > cut)) continue;
        double proj = 0.0;
        for (int i = 0; i < m; ++i) proj += V[i * m + k];
        proj /= lam;
        for (int i = 0; i < m; ++i) x[i] += proj * V[i * m + k];
    }
}

// Index of pair (p, q), p <= q, in the row-major upper triangle of an m x m
// symmetric matrix.
__host__ __device__ constexpr int aa_pair(int p, int q, int m) {
    return p * m - (p * (p - 1)) / 2 + (q - p);
}
// Pair t of the same order.
__device__ __forceinline__ void aa_pair_of(int t, int m, int& p, int& q) {
    p = 0;
    while (t >= m - p) {
        t -= m - p;
        ++p;
    }
    q = p + t;
}
__device__ __forceinline__ double aa_clip(double a, double alpha_max) {
    if (alpha_max > 0.0) {
        if (a < -alpha_max) a = -alpha_max;
        if (a > alpha_max) a = alpha_max;
    }
    return a;
}

// Anderson coefficients for a history of compile-time length M in one thread,
// the factor in registers: (G + reg I) x = 1 by Cholesky with the sums in the
// order of aa_small_solve, then alpha = x / sum(x), clipped
// (bgk1d_aa_cpu.py:146-168).  Each pivot is kept as its reciprocal square
// root and the divisions by it are multiplications, so the dependent chain of
// a column is one rsqrt.  False (nothing written) when a pivot is not
// positive, for the min-norm fall-back.
template <int M>
__device__ __forceinline__ bool aa_alpha_fixed(const double* gs, double reg, double alpha_max,
                                               double* alpha_out) {
    double L[M][M], rd[M];  // strict lower factor; rd[j] = 1 / L[j][j]
#pragma unroll
    for (int i = 0; i < M; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) L[i][j] = gs[aa_pair(j, i, M)] + (i == j ? reg : 0.0);
#pragma unroll
    for (int j = 0; j < M; ++j) {
        double s = L[j][j];
#pragma unroll
        for (int k = 0; k < j; ++k) s -= L[j][k] * L[j][k];
        if (!(s > 0.0)) return false;
        rd[j] = rsqrt(s);
#pragma unroll
        for (int i = j + 1; i < M; ++i) {
            double t = L[i][j];
#pragma unroll
            for (int k = 0; k < j; ++k) t -= L[i][k] * L[j][k];
            L[i][j] = t * rd[j];
        }
    }
    double y[M], x[M];
#pragma unroll
    for (int i = 0; i < M; ++i) {
        double t = 1.0;
#pragma unroll
        for (int k = 0; k < i; ++k) t -= L[i][k] * y[k];
        y[i] = t * rd[i];
    }
#pragma unroll
    for (int i = M - 1; i >= 0; --i) {
        double t = y[i];
#pragma unroll
        for (int k = i + 1; k < M; ++k) t -= L[k][i] * x[k];
        x[i] = t * rd[i];
    }
    double asum = 0.0;
#pragma unroll
    for (int p = 0; p < M; ++p) asum += x[p];
    if (fabs(asum) < 1.0e-30) asum = 1.0e-30;
    const double rs = 1.0 / asum;
#pragma unroll
    for (int p = 0; p < M; ++p) alpha_out[p] = aa_clip(x[p] * rs, alpha_max);
    return true;
}

// Gram matrix entries of four pairs from the blocks' partials (one warp): lane
// l sums blocks l, l+32, ..., then a butterfly.
__device__ __forceinline__ void aa_pair_sums(const double* const (&g)[4], int nblk, double (&v)[4]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = 0.0;
    for (int r0 = 0; r0 < nblk; r0 += 160) {
        double t[4][5];
#pragma unroll
        for (int c = 0; c < 5; ++c) {  // clamped: every load is issued
            const int r = r0 + 32 * c + lane < nblk ? r0 + 32 * c + lane : nblk - 1;
#pragma unroll
            for (int u = 0; u < 4; ++u) t[u][c] = ld_cg(&g[u][r]);
        }
#pragma unroll
        for (int c = 0; c < 5; ++c)
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] += r0 + 32 * c + lane < nblk ? t[u][c] : 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] += __shfl_xor_sync(0xffffffffu, v[u], o);
}

__device__ __forceinline__ double div_signed(double a, double d) {
    return d < 0.0 ? -div_nr(a, -d) : div_nr(a, d);
}

// Anderson coefficients by one warp: (G + reg I) x = 1 by Gauss-Jordan
// elimination without pivoting (lane i holds row i; the pivots are those of
// the Cholesky factorisation, whose failure is a pivot that is not positive),
// alpha = x / sum(x), clipped (bgk1d_aa_cpu.py:146-168).  gs: the pairs
// p <= q row by row.  Lane j < mh returns alpha_j.  About 260 cycles a column;
// the single-lane Cholesky with its two substitutions took three times that.
// gram(p, q): entry of the columns p and q.
template <class Gram>
__device__ __forceinline__ double aa_solve_gram(Gram gram, int mh, double reg, double alpha_max) {
    const int lane = threadIdx.x & 31;
    double row[kMaxAACols], rhs = 1.0, rinv = 0.0;
    const int i = lane < mh ? lane : mh - 1;
#pragma unroll
    for (int j = 0; j < kMaxAACols; ++j) {
        const int jc = j < mh ? j : mh - 1;
        row[j] = gram(i, jc) + (j == i ? reg : 0.0);
    }
    bool ok = true;
#pragma unroll
    for (int k = 0; k < kMaxAACols; ++k) {
        if (k >= mh) break;
        const double pk = __shfl_sync(0xffffffffu, row[k], k);
        if (!(pk > 0.0)) {
            ok = false;
            break;
        }
        const double r = pk >= 1e-270 && pk <= 1e270 ? recip3(pk) : 1.0 / pk;
        if (lane == k) rinv = r;
        const double f = lane == k ? 0.0 : row[k] * r;
#pragma unroll
        for (int j = k + 1; j < kMaxAACols; ++j)
            row[j] = fma(-f, __shfl_sync(0xffffffffu, row[j], k), row[j]);
        rhs = fma(-f, __shfl_sync(0xffffffffu, rhs, k), rhs);
    }
    double x = rhs * rinv;
    if (!ok) {
        // not positive definite: the min-norm fall-back on the full matrix, by one
        // lane (32 lanes with arrays of their own take a third longer)
        double A[kMaxAACols * kMaxAACols], xv[kMaxAACols];
        if (lane == 0) {
            for (int p = 0; p < mh; ++p)
                for (int q = 0; q < mh; ++q) A[p * mh + q] = gram(p, q) + (p == q ? reg : 0.0);
            aa_small_solve(mh, A, xv);
        }
        __syncwarp();
        for (int p = 0; p < mh; ++p) {
            const double t = __shfl_sync(0xffffffffu, lane == 0 ? xv[p] : 0.0, 0);
            x = i == p ? t : x;
        }
    }
    double asum = 0.0;
    for (int p = 0; p < mh; ++p) asum += __shfl_sync(0xffffffffu, x, p);
    if (fabs(asum) < 1.0e-30) asum = 1.0e-30;
    return aa_clip(div_signed(x, asum), alpha_max);
}
static __device__ __noinline__ double aa_solve_warp(const double* gs, int mh, double reg, double alpha_max) {
    return aa_solve_gram([&](int p, int q) { return gs[aa_pair(p < q ? p : q, p < q ? q : p, mh)]; }, mh, reg,
                         alpha_max);
}

// Last reduction block of Anderson call m: Gram matrix from the per-block
// partials, stored pair-major (lane l sums blocks l, l+32, ... of eight pairs
// at a time, 32 loads in flight, then a butterfly over the lanes; the sums go
// through the warp's scratch `gs` in shared memory),
// regularised Cholesky solve, normalisation by the sum, clip
// (bgk1d_aa_cpu.py:146-168).
static __device__ __noinline__ void aa_finalize(const double* gpart, int nrb, int mh, double reg,
                                         double alpha_max, double* alpha_out, double* gs) {
    const int lane = threadIdx.x & 31;
    const int npairs = mh * (mh + 1) / 2;
    for (int q0 = 0; q0 < npairs; q0 += 8) {
        double acc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc[u] = 0.0;
        for (int r0 = 0; r0 < nrb; r0 += 128) {
            double t[8][4];
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    // clamped indices: every load is issued, the extra ones add 0
                    const int r = r0 + 32 * c + lane;
                    const bool in = q0 + u < npairs && r < nrb;
                    const int qc = q0 + u < npairs ? q0 + u : npairs - 1;
                    const double v = ld_cg(&gpart[(size_t)qc * nrb + (r < nrb ? r : nrb - 1)]);
                    t[u][c] = in ? v : 0.0;
                }
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[u] += t[u][c];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) acc[u] = warp_sum(acc[u]);
        if (lane == 0)
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (q0 + u < npairs) gs[q0 + u] = acc[u];
    }
    __syncwarp();
    if (lane != 0) return;
    bool ok = false;
    switch (mh) {
        case 1: ok = aa_alpha_fixed<1>(gs, reg, alpha_max, alpha_out); break;
        case 2: ok = aa_alpha_fixed<2>(gs, reg, alpha_max, alpha_out); break;
        case 3: ok = aa_alpha_fixed<3>(gs, reg, alpha_max, alpha_out); break;
        case 4: ok = aa_alpha_fixed<4>(gs, reg, alpha_max, alpha_out); break;
        case 5: ok = aa_alpha_fixed<5>(gs, reg, alpha_max, alpha_out); break;
        case 6: ok = aa_alpha_fixed<6>(gs, reg, alpha_max, alpha_out); break;
        case 7: ok = aa_alpha_fixed<7>(gs, reg, alpha_max, alpha_out); break;
        default: ok = aa_alpha_fixed<8>(gs, reg, alpha_max, alpha_out); break;
    }
    if (ok) return;
    // not positive definite: the min-norm fall-back on the full matrix
    double A[kMaxAACols * kMaxAACols], xv[kMaxAACols];
    for (int p = 0; p < mh; ++p)
        for (int q = 0; q < mh; ++q) {
            const int a = p < q ? p : q, b = p < q ? q : p;
            A[p * mh + q] = gs[aa_pair(a, b, mh)] + (p == q ? reg : 0.0);
        }
    aa_small_solve(mh, A, xv);
    double asum = 0.0;
    for (int p = 0; p < mh; ++p) asum += xv[p];
    if (fabs(asum) < 1.0e-30) asum = 1.0e-30;
    for (int p = 0; p < mh; ++p) alpha_out[p] = aa_clip(xv[p] / asum, alpha_max);
}

// Phase trace (off unless a buffer is attached): per Picard iteration the
// earliest start and latest end over all warps of the pass, in
// %globaltimer nanoseconds: [m][0] min start, [1] max end; [2], [3] unused.
constexpr int kTracePhases = 4;
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void trace_mark(const PlanDev& P, int m, int ph, bool is_min) {
    if (P.head.trace == nullptr || (threadIdx.x & 31) != 0 || m >= P.head.trace_iters) return;
    unsigned long long* slot = P.head.trace + (size_t)m * kTracePhases + ph;
    const unsigned long long t = gtimer();
    if (is_min) atomicMin(slot, t); else atomicMax(slot, t);
}

// Grid barrier of a launch; on a timeout the error is also recorded in the
// sticky word read by keq_plan_error.
__device__ __forceinline__ bool plan_sync(PlanDev& P, unsigned G) {
    if (grid_sync(&P.head.bar, G, &P.head.err, P.head.spin_limit)) return true;
    if (threadIdx.x == 0) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
    return false;
}

}  // namespace keq
