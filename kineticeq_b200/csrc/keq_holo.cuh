// keq_holo.cuh -- what the two HOLO step kernels share: the instance and plan
// records, the moment formulas, the low-order (LO) block rows and their
// solution by parallel cyclic reduction.
//   keq_holo.cu       tiles with a decoupled look-back, any size; plan construction
//   keq_holo_rows.cu  row blocks owned by one CTA, without grid barriers
#pragma once

#include "keq_common.cuh"
#include "keq_internal.h"
#include "keq_tile.cuh"

namespace keq {
namespace holo {

constexpr double kTheta = 0.5;
constexpr int kLoChunk = 32;        // rows per LO chunk (one per lane)
constexpr int kMaxLoChunks = 512;   // LO chunks per instance at most (16 groups of 32)

struct HoloInst {
    int nx, nv, n_inner, kp;
    int nt_neg, nvt, nchunks, nrb;
    int rows, lo_len, lo_k, pad0;  // tile rows; LO chunk length and count
    long long tile_off, rb_off, lo_off;
    double dx, dv, dt, tau_tilde, dtdx2;  // dtdx2 = dt / (2 dx)
    int ho_iter, lo_iter, con_terms, flux_cons;
    int sv_down, fixed_ho, fixed_lo, pad1;
    double ho_tol, ho_abs_tol, lo_tol, lo_abs_tol;
    const double* v;
    const double* f_in;
    double* f_out;
    keq_step_stats* stats;
    // workspace carve
    double* E;       // nx*nv : explicit term (interior rows)
    double* part;    // nvt*n_inner*kPartQ : moment / Maxwellian partials
    double* R;       // nx*8 : raw half-range sums of f_z (v>0: 1,v,v^2,v^3 | v<=0: same)
    double* Rn;      // nx*8 : same for f^n
    double* Mco;     // nx*4 : HO-old (u, -0.5/T, n/sqrt(2 pi T), 1/tau)
    double* Wm;      // nx*3 : LO iterate W_m = (n, nu, U)
    double* Who;     // nx*3 : W_HO
    double* Iold;    // nx*3 : old collision moments (1-theta) C_old . w dv
    double* Msum;    // nx*3 : velocity sums of M(f_z) per row: sum M, sum M v, sum M v^2 / 2
    double* Ib;      // 8    : boundary-row Maxwellian sums (2 rows x 3) + spare
    double* Y;       // nx*3 : consistency terms of the current HO iteration
    double* T1;      // nx*3 : W_HO - dt/2dx (F_HO diff) of the current HO iteration
    double* lorow;   // 2*n_inner*13 : y(3) | P(2x2) | P_U | Q(2x2) | Q_U per row, one set per
                     // LO-iteration parity (iteration m writes set m & 1)
    double* loedge;  // lo_k*18 : last-row blocks of each chunk (A,B,C 2x2, D 2 | U: a,b,c,d)
    double* xi;      // lo_k*3 : interface unknowns
    double* Wlo;     // 3*nx : n_lo | u_lo | T_lo of the last LO solve (state.n/u/T)
    double* agg;     // ntiles*64 : tile maps (distribution pass)
    double* inc;     // ntiles*32 : tile carries
    unsigned long long* flag;  // ntiles : look-back flags
    unsigned* rbcnt; // ho_iter*nrb : row-block arrivals of the distribution pass
    double* ho_red;  // ho_iter*4 : HO std residual, max |df|, max ref, max |Y|
    double* lo_hist; // ho_iter*lo_iter*2 : LO max |dW|, std residual
    int* ho_run;     // ho_iter : 1 if HO iteration z ran
    int* lo_run;     // ho_iter*lo_iter : 1 if LO iteration m of HO iteration z ran
    int* nonfin;     // ho_iter : non-finite flag of f_{z+1}
    // row-block kernel (keq_holo_rows.cu, keq_rows.cuh)
    int rblk, nblk, kmax, lo_n;  // rows per block, blocks, blocks of a fold at most, LO chunks
    double* xin;        // nblk*nvt*32 : inflow of each block's tiles in the last sweep
    ulonglong2* maps;   // nblk * nvt * 64 : block maps (published behind the HO residuals of all blocks)
    ulonglong2* horec;  // 2 * nblk * 4 : HO residuals of the blocks
    ulonglong2* rowd;   // nx * 12 : raw half-range sums (8) and Maxwellian sums (3) of f_z per row
    ulonglong2* lorec;  // 2 * lo_n * 40 : LO chunks' interface data and residuals
    ulonglong2* lowx;   // 2 * n_inner * 3 : LO iterate of the rows
    ulonglong2* lores;  // 4 * 2 * lo_n : LO residuals (negative: flag) and differences of the chunks
    ulonglong2* locm;   // lo_n : the chunks' largest Maxwellian coefficient
    ulonglong2* loy;    // lo_n : the chunks' largest |Y|
    ulonglong2* wlo;    // nx * 4 : LO solution (n, nu, U)
    double* misc;    // 8 : [0] max |f^n| over the boundary rows, [1] max |Y| of the boundary rows, [2] max |E|
                     // (row-block kernel: two sets of 4 by launch parity)
};

struct HoloDev {
    PlanHead head;
    long long* blk_off;  // row-block kernel: n_inst+1
    int n_inst;
    int max_ho, max_lo;
    int pad;
    long long total_tiles, total_rb, total_lo;
    HoloInst* inst;
    long long* tile_off;
    long long* rb_off;
    long long* lo_off;
    unsigned* tickets;  // max_ho : tile claims of the distribution pass
    unsigned long long arrivals;  // row-block kernel: launch_barrier
};

// Phase trace (off unless a buffer is attached): four rows of 4 stamps
// (%globaltimer ns) per HO iteration z:
//   row 4z   = [A start (min), A work end (max), LO start (min), LO end (max)]
//   row 4z+1 = [C start (min), C work end (max), LO iterations, 0]
// and of the look-back kernel
//   row 4z+2 = LO iteration 0: [L1 start (min), L1 end (max), L2 start (min), L2 end (max)]
//   row 4z+3 = LO iteration 0: [L3 start (min), L3 end (max), after its barrier (min), 0]
// or of the row-block kernel
//   row 4z+2 = [LO solve in the chunks' CTAs start (min), end (max),
//               wait for its solution start (min), end (max)]
//   row 4z+3 = [HO residual exchange start (min), end (max), UINT64_MAX, 0]
__device__ __forceinline__ unsigned long long gtimer_h() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void trace_h(const HoloDev& P, int z, int slot, bool is_min) {
    if (P.head.trace == nullptr || (threadIdx.x & 31) != 0 || 4 * z + 3 >= P.head.trace_iters)
        return;
    unsigned long long* p = P.head.trace + (size_t)16 * z + slot;
    const unsigned long long t = gtimer_h();
    if (is_min) atomicMin(p, t); else atomicMax(p, t);
}

// LO chunk scratch (per warp, aliasing the tile buffers of WarpSmem).
struct LoRow {
    double A[4], B[4], C[4], D[2];  // (n, nu) blocks, row-major 2x2
    double a, b, c, d;              // U
    double cu;                      // U: C' of the forward sweep
};

// calculate_moments (bgk1d_utils/general/bgk1d_compute_moments.py:7-17) from
// raw half-range sums: n = sum f dv, u = (sum f v dv)/n, T = (sum f v^2 dv)/n - u^2.
struct Mom {
    double n, u, T, s1, s2, s3;  // s_k = sum f v^k dv
};
__device__ __forceinline__ Mom mom_of(const double* R8, double dv) {
    Mom m;
    m.n = (R8[0] + R8[4]) * dv;
    m.s1 = (R8[1] + R8[5]) * dv;
    m.s2 = (R8[2] + R8[6]) * dv;
    m.s3 = (R8[3] + R8[7]) * dv;
    m.u = m.s1 / m.n;
    m.T = m.s2 / m.n - m.u * m.u;
    return m;
}
// Q = 1/2 sum (v-u)^3 f dv (_HO_calculate_fluxes_Q, :81-99) by the binomial
// expansion of the raw moments.
__device__ __forceinline__ double q_of(const Mom& m) {
    const double u = m.u;
    return 0.5 * (m.s3 - 3.0 * u * m.s2 + 3.0 * u * u * m.s1 - u * u * u * m.n);
}

// Maxwellian coefficients of (n, u, T) (bgk1d_maxwellian.py:7-33) and 1/tau.
__device__ __forceinline__ void mc_of(const Mom& m, double tau_tilde, double* c4) {
    const double sT = sqrt(m.T);
    c4[0] = m.u;
    c4[1] = -(0.5 / m.T);
    c4[2] = (m.n * kInvSqrt2Pi) / sT;
    c4[3] = (m.n * sT) / tau_tilde;  // 1/tau, tau = tau_tilde / (n sqrt(T))
}

// Sum over the velocities of a Maxwellian times (1, v, v^2/2), one warp.
__device__ __forceinline__ void maxwell_sums_row(const double* v, int nv, const double* c4,
                                                 double* s3) {
    const int lane = threadIdx.x & 31;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    for (int j = lane; j < nv; j += 32) {
        const double vj = __ldg(&v[j]);
        const double d = vj - c4[0];
        const double M = c4[2] * exp_nonpos(d * d * c4[1]);
        a0 += M;
        a1 += M * vj;
        a2 += M * vj * vj;
    }
    s3[0] = warp_sum(a0);
    s3[1] = warp_sum(a1);
    s3[2] = 0.5 * warp_sum(a2);
}

// ---- LO: structured blocks -----------------------------------------------------
// u*, P* of a cell from W = (n, nu, U) (:293-303): den = n + 1e-30,
// u = nu/den, T = max(2 (U/den - u^2/2), 1e-30), P = n T.
// kShort: with the short division.
template <bool kShort>
__device__ __forceinline__ void star_of(const double* W3, double& us, double& Ps) {
    const double den = W3[0] + 1e-30;
    us = kShort ? div_nr(W3[1], den) : W3[1] / den;
    double Ts = 2.0 * ((kShort ? div_nr(W3[2], den) : W3[2] / den) - 0.5 * us * us);
    Ts = (Ts != Ts || Ts >= 1e-30) ? Ts : 1e-30;
    Ps = W3[0] * Ts;
}

// 1/d for |d| >= 1e-30: the short form (recip3) where it is valid.  A division
// is about 700 cycles of latency, and every PCR step starts with two.
__device__ __forceinline__ double rcp_fast(double d) {
    return fabs(d) <= 1e270 ? recip3(d) : 1.0 / d;
}
__device__ __forceinline__ bool inv2(const double* M, double* Mi) {
    const double det = M[0] * M[3] - M[1] * M[2];
    if (!(fabs(det) >= 1e-30)) {
        Mi[0] = Mi[1] = Mi[2] = Mi[3] = 0.0;
        return false;
    }
    const double id = rcp_fast(det);
    Mi[0] = M[3] * id;
    Mi[1] = -M[1] * id;
    Mi[2] = -M[2] * id;
    Mi[3] = M[0] * id;
    return true;
}
__device__ __forceinline__ void mm2(const double* A, const double* B, double* C) {
    C[0] = A[0] * B[0] + A[1] * B[2];
    C[1] = A[0] * B[1] + A[1] * B[3];
    C[2] = A[2] * B[0] + A[3] * B[2];
    C[3] = A[2] * B[1] + A[3] * B[3];
}
__device__ __forceinline__ void mv2(const double* A, const double* x, double* y) {
    y[0] = A[0] * x[0] + A[1] * x[1];
    y[1] = A[2] * x[0] + A[3] * x[1];
}
__device__ __forceinline__ double rcp_or0(double d) { return fabs(d) >= 1e-30 ? rcp_fast(d) : 0.0; }

// Block row of interior row k (cell i = k+1) from W_m: faces L (i-1, i) and
// R (i, i+1); AA = -c4 A_L (0 at k = 0), CC = c4 A_R (0 at the last row),
// BB = I + c4 (A_R - A_L), DD = ((T1 - c2 (b_R - b_L)) + Y).
template <bool kShort = false>
__device__ __forceinline__ void lo_row_w(const HoloInst& I, int k, const double* Wl,
                                         const double* Wc, const double* Wr, const double* T1,
                                         const double* Y, LoRow& r) {
    double uL, PL, uC, PC, uR, PR;
    star_of<kShort>(Wl, uL, PL);
    star_of<kShort>(Wc, uC, PC);
    star_of<kShort>(Wr, uR, PR);
    const double uhL = 0.5 * (uL + uC), PhL = 0.5 * (PL + PC);
    const double uhR = 0.5 * (uC + uR), PhR = 0.5 * (PC + PR);
    // (dt / (4 dx) and dt / (2 dx), exactly)
    const double c4 = 0.5 * I.dtdx2, c2 = I.dtdx2;
    const double aL = (k >= 1) ? 1.0 : 0.0, aR = (k <= I.n_inner - 2) ? 1.0 : 0.0;
    // A_int = [[0,1,0],[uh^2,0,0],[0,0,uh]]
    const double uL2 = uhL * uhL, uR2 = uhR * uhR;
    r.A[0] = 0.0; r.A[1] = aL * (1.0 * (-c4)); r.A[2] = aL * (uL2 * (-c4)); r.A[3] = 0.0;
    r.C[0] = 0.0; r.C[1] = aR * (1.0 * c4); r.C[2] = aR * (uR2 * c4); r.C[3] = 0.0;
    r.B[0] = (0.0 - 0.0) * c4 + 1.0;
    r.B[1] = (1.0 - 1.0) * c4;
    r.B[2] = (uR2 - uL2) * c4;
    r.B[3] = (0.0 - 0.0) * c4 + 1.0;
    r.a = aL * (uhL * (-c4));
    r.c = aR * (uhR * c4);
    r.b = (uhR - uhL) * c4 + 1.0;
    // b_int = (0, Ph, uh Ph)
    const double bd0 = 0.0 - 0.0, bd1 = PhR - PhL, bd2 = uhR * PhR - uhL * PhL;
    r.D[0] = __dadd_rn(__dadd_rn(T1[0], __dmul_rn(-c2, bd0)), Y[0]);
    r.D[1] = __dadd_rn(__dadd_rn(T1[1], __dmul_rn(-c2, bd1)), Y[1]);
    r.d = __dadd_rn(__dadd_rn(T1[2], __dmul_rn(-c2, bd2)), Y[2]);
}

// ---- LO: warp-parallel block PCR ---------------------------------------------
// One block row per lane of a block-tridiagonal system with 2x2 blocks for
// (n, nu) and a scalar system for U:
//     A x_{l-1} + B x_l + C x_{l+1} = R,   a u_{l-1} + b u_l + c u_{l+1} = r,
// R holding 5 right-hand-side columns (2 x 5, row-major) and r 3.  Parallel
// cyclic reduction over the lanes: at stride d every row eliminates its
// couplings to rows l-d and l+d with their (pre-step) blocks, fetched by
// shuffles; after log2(L) steps every row is decoupled and B^{-1} R, r / b
// are the solution columns.  Lanes >= L carry identity rows.
struct PcrRow {
    double A[4], B[4], C[4], R[10];
    double a, b, c, r[3];
};

__device__ __forceinline__ double shup(double v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ double shdn(double v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }

__device__ __forceinline__ void identity_row(PcrRow& q) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        q.A[k] = 0.0;
        q.C[k] = 0.0;
        q.B[k] = (k == 0 || k == 3) ? 1.0 : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 10; ++k) q.R[k] = 0.0;
    q.a = 0.0; q.b = 1.0; q.c = 0.0;
    q.r[0] = q.r[1] = q.r[2] = 0.0;
}

__device__ __forceinline__ void warp_pcr(PcrRow& q, int L) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int d = 1; d < L; d <<= 1) {
        double Bi[4];
        inv2(q.B, Bi);
        const double bi = rcp_or0(q.b);
        // Early exit once every row is decoupled to below double rounding:
        // |B^{-1}|_inf (|A|_inf + |C|_inf) <= 2^-60 and the same for the
        // scalar rows.  The couplings of an interface system are products of
        // a chunk's 31 row couplings, so this usually holds before the first
        // step there.  The test is warp-uniform and depends on the data only.
        {
            const double nbi = fmax(fabs(Bi[0]) + fabs(Bi[1]), fabs(Bi[2]) + fabs(Bi[3]));
            const double nac = fmax(fabs(q.A[0]) + fabs(q.A[1]), fabs(q.A[2]) + fabs(q.A[3])) +
                               fmax(fabs(q.C[0]) + fabs(q.C[1]), fabs(q.C[2]) + fabs(q.C[3]));
            const double kTiny = 8.673617379884035e-19;  // 2^-60
            const bool dec = nbi * nac <= kTiny && fabs(bi) * (fabs(q.a) + fabs(q.c)) <= kTiny;
            if (__all_sync(0xffffffffu, dec || lane >= L)) break;
        }
        const bool has_lo = lane >= d && lane < L, has_hi = lane + d < L;
        double nA[4], nC[4], dB[4], nR[10];
        double na, nc, db, nr[3];
        // lower neighbour: alpha = -A B_lo^{-1}
        {
            double t[4], al[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = shup(Bi[k], d);
            mm2(q.A, t, al);
#pragma unroll
            for (int k = 0; k < 4; ++k) al[k] = has_lo ? -al[k] : 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = shup(q.A[k], d);
            mm2(al, t, nA);
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = shup(q.C[k], d);
            mm2(al, t, dB);
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const double r0 = shup(q.R[j], d), r1 = shup(q.R[5 + j], d);
                nR[j] = q.R[j] + (al[0] * r0 + al[1] * r1);
                nR[5 + j] = q.R[5 + j] + (al[2] * r0 + al[3] * r1);
            }
            const double bl = shup(bi, d);  // every lane shuffles; the mask is the full warp
            const double a1 = has_lo ? -q.a * bl : 0.0;
            na = a1 * shup(q.a, d);
            db = a1 * shup(q.c, d);
#pragma unroll
            for (int j = 0; j < 3; ++j) nr[j] = q.r[j] + a1 * shup(q.r[j], d);
        }
        // upper neighbour: gamma = -C B_hi^{-1}
        {
            double t[4], ga[4], u[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = shdn(Bi[k], d);
            mm2(q.C, t, ga);
#pragma unroll
            for (int k = 0; k < 4; ++k) ga[k] = has_hi ? -ga[k] : 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = shdn(q.C[k], d);
            mm2(ga, t, nC);
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = shdn(q.A[k], d);
            mm2(ga, t, u);
#pragma unroll
            for (int k = 0; k < 4; ++k) dB[k] += u[k];
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const double r0 = shdn(q.R[j], d), r1 = shdn(q.R[5 + j], d);
                nR[j] += ga[0] * r0 + ga[1] * r1;
                nR[5 + j] += ga[2] * r0 + ga[3] * r1;
            }
            const double bh = shdn(bi, d);
            const double g1 = has_hi ? -q.c * bh : 0.0;
            nc = g1 * shdn(q.c, d);
            db += g1 * shdn(q.a, d);
#pragma unroll
            for (int j = 0; j < 3; ++j) nr[j] += g1 * shdn(q.r[j], d);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            q.A[k] = nA[k];
            q.C[k] = nC[k];
            q.B[k] += dB[k];
        }
#pragma unroll
        for (int k = 0; k < 10; ++k) q.R[k] = nR[k];
        q.a = na;
        q.c = nc;
        q.b += db;
#pragma unroll
        for (int j = 0; j < 3; ++j) q.r[j] = nr[j];
    }
    double Bi[4];
    inv2(q.B, Bi);
    double nR[10];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        nR[j] = Bi[0] * q.R[j] + Bi[1] * q.R[5 + j];
        nR[5 + j] = Bi[2] * q.R[j] + Bi[3] * q.R[5 + j];
    }
#pragma unroll
    for (int k = 0; k < 10; ++k) q.R[k] = nR[k];
    const double bi = rcp_or0(q.b);
#pragma unroll
    for (int j = 0; j < 3; ++j) q.r[j] *= bi;
}

// Solution columns [y | P | Q] of a PCR row as the 13-value representation
// y(2) y_U | P(2x2) P_U | Q(2x2) Q_U of x = y + P x_left + Q x_right.
__device__ __forceinline__ void rep_of(const PcrRow& q, double* o) {
    o[0] = q.R[0]; o[1] = q.R[5]; o[2] = q.r[0];
    o[3] = q.R[1]; o[4] = q.R[2]; o[5] = q.R[6]; o[6] = q.R[7]; o[7] = q.r[1];
    o[8] = q.R[3]; o[9] = q.R[4]; o[10] = q.R[8]; o[11] = q.R[9]; o[12] = q.r[2];
}

// Local system of L rows (lane l = row l, couplings A_l, C_l) with the
// left coupling of row 0 and the right coupling of row L-1 moved to the
// right-hand side as the P and Q columns (D, -A_0 e_0, -C_{L-1} e_{L-1}).
__device__ __forceinline__ void local_rows(PcrRow& q, const double* A, const double* B,
                                           const double* C, const double* D, double a, double b,
                                           double c, double d, int l, int L) {
    if (l >= L) {
        identity_row(q);
        return;
    }
    const bool first = l == 0, last = l == L - 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        q.A[k] = first ? 0.0 : A[k];
        q.B[k] = B[k];
        q.C[k] = last ? 0.0 : C[k];
    }
    q.R[0] = D[0];
    q.R[5] = D[1];
    q.R[1] = first ? -A[0] : 0.0; q.R[2] = first ? -A[1] : 0.0;
    q.R[6] = first ? -A[2] : 0.0; q.R[7] = first ? -A[3] : 0.0;
    q.R[3] = last ? -C[0] : 0.0; q.R[4] = last ? -C[1] : 0.0;
    q.R[8] = last ? -C[2] : 0.0; q.R[9] = last ? -C[3] : 0.0;
    q.a = first ? 0.0 : a;
    q.b = b;
    q.c = last ? 0.0 : c;
    q.r[0] = d;
    q.r[1] = first ? -a : 0.0;
    q.r[2] = last ? -c : 0.0;
}

// L2: the interface system of the K = lo_k chunks, one CTA per instance.
// The interface rows are split into groups of 32; each group is solved by
// warp PCR into xi_k = y_k + P_k X_{g-1} + Q_k X_g in terms of the group
// interfaces X_g (the last interface of every group), whose own system (at
// most 32 unknowns) is solved by warp 0 the same way; then every xi_k is
// recovered into I.xi.
struct GroupRec {
    double rep_prev[13];  // representation of the group row before the last
    double rep_first[13]; // representation of the group's first row
    double al[4], be[4], ga[4], de[2], s4[4];  // the group's last interface row
};

template <class RowLoad, class Store>
__device__ __forceinline__ void lo_reduced_solve(int K, unsigned char* smem, RowLoad row, Store store) {
    const int G = (K + 31) / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    GroupRec* grec = reinterpret_cast<GroupRec*>(smem);
    double* reps = reinterpret_cast<double*>(smem + sizeof(GroupRec) * G);  // K x 13
    double* X = reps + 13 * (size_t)K;                                      // G x 3
    for (int g = warp; g < G; g += (int)(blockDim.x >> 5)) {
        const int k0 = 32 * g;
        const int len = (K - k0) < 32 ? (K - k0) : 32;
        const int nloc = len - 1;
        const int k = k0 + lane;
        double al[4] = {0, 0, 0, 0}, be[4] = {1, 0, 0, 1}, ga[4] = {0, 0, 0, 0}, de[2] = {0, 0};
        double s4[4] = {0.0, 1.0, 0.0, 0.0};
        if (lane < len) row(k, al, be, ga, de, s4);
        PcrRow q;
        local_rows(q, al, be, ga, de, s4[0], s4[1], s4[2], s4[3], lane, nloc);
        warp_pcr(q, nloc);
        double o[13];
        if (lane < nloc) {
            rep_of(q, o);
        } else {
#pragma unroll
            for (int t = 0; t < 13; ++t) o[t] = 0.0;
            o[8] = 1.0; o[11] = 1.0; o[12] = 1.0;
        }
        if (lane < len) {
#pragma unroll
            for (int t = 0; t < 13; ++t) reps[13 * (size_t)k + t] = o[t];
        }
        if (lane == nloc) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                grec[g].al[t] = al[t];
                grec[g].be[t] = be[t];
                grec[g].ga[t] = ga[t];
                grec[g].s4[t] = s4[t];
            }
            grec[g].de[0] = de[0];
            grec[g].de[1] = de[1];
        }
        __syncwarp();
        if (lane < 13) {
            grec[g].rep_first[lane] = reps[13 * (size_t)k0 + lane];
            grec[g].rep_prev[lane] = (nloc >= 1) ? reps[13 * (size_t)(k0 + nloc - 1) + lane]
                                                 : ((lane == 3 || lane == 6 || lane == 7) ? 1.0 : 0.0);
        }
    }
    __syncthreads();
    // group interfaces: the same interface-row construction one level up
    if (warp == 0) {
        double A[4] = {0, 0, 0, 0}, B[4] = {1, 0, 0, 1}, C[4] = {0, 0, 0, 0}, D[2] = {0, 0};
        double a = 0.0, b = 1.0, c = 0.0, d = 0.0;
        if (lane < G) {
            const GroupRec& gr = grec[lane];
            const double* pm = gr.rep_prev;
            double nx_[13];
#pragma unroll
            for (int t = 0; t < 13; ++t) nx_[t] = (lane + 1 < G) ? grec[lane + 1].rep_first[t] : 0.0;
            double T4[4], U4[4], t2[2], u2[2];
            mm2(gr.al, pm + 3, A);
            mm2(gr.al, pm + 8, T4);
            mm2(gr.ga, nx_ + 3, U4);
#pragma unroll
            for (int t = 0; t < 4; ++t) B[t] = gr.be[t] + T4[t] + U4[t];
            mm2(gr.ga, nx_ + 8, C);
            mv2(gr.al, pm, t2);
            mv2(gr.ga, nx_, u2);
            D[0] = gr.de[0] - t2[0] - u2[0];
            D[1] = gr.de[1] - t2[1] - u2[1];
            a = gr.s4[0] * pm[7];
            b = gr.s4[1] + gr.s4[0] * pm[12] + gr.s4[2] * nx_[7];
            c = gr.s4[2] * nx_[12];
            d = gr.s4[3] - gr.s4[0] * pm[2] - gr.s4[2] * nx_[2];
        }
        PcrRow q;
        if (lane < G) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                q.A[t] = A[t];
                q.B[t] = B[t];
                q.C[t] = C[t];
            }
#pragma unroll
            for (int t = 0; t < 10; ++t) q.R[t] = 0.0;
            q.R[0] = D[0];
            q.R[5] = D[1];
            q.a = a; q.b = b; q.c = c;
            q.r[0] = d; q.r[1] = 0.0; q.r[2] = 0.0;
        } else {
            identity_row(q);
        }
        warp_pcr(q, G);
        if (lane < G) {
            X[3 * lane + 0] = q.R[0];
            X[3 * lane + 1] = q.R[5];
            X[3 * lane + 2] = q.r[0];
        }
    }
    __syncthreads();
    // every interface unknown from its group representation
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        const int g = k >> 5;
        const double* o = reps + 13 * (size_t)k;
        double xl[3] = {0.0, 0.0, 0.0};
        if (g > 0)
#pragma unroll
            for (int t = 0; t < 3; ++t) xl[t] = X[3 * (g - 1) + t];
        const double xr[3] = {X[3 * g], X[3 * g + 1], X[3 * g + 2]};
        double x0 = o[0] + (o[3] * xl[0] + o[4] * xl[1]) + (o[8] * xr[0] + o[9] * xr[1]);
        double x1 = o[1] + (o[5] * xl[0] + o[6] * xl[1]) + (o[10] * xr[0] + o[11] * xr[1]);
        double x2 = o[2] + o[7] * xl[2] + o[12] * xr[2];
        store(k, x0, x1, x2);
    }
    __syncthreads();
}

// x = y + P xl + Q xr for a row with representation o (13 values), in one
// fixed, non-contracted order: a chunk's warp recovers its rows with it, and
// the previous chunk's warp recomputes this chunk's first row with it, so
// both get the same value.
__device__ __forceinline__ void rep_apply(const double* o, const double* xl, const double* xr,
                                          double* x) {
    x[0] = __dadd_rn(__dadd_rn(o[0], __dadd_rn(__dmul_rn(o[3], xl[0]), __dmul_rn(o[4], xl[1]))),
                     __dadd_rn(__dmul_rn(o[8], xr[0]), __dmul_rn(o[9], xr[1])));
    x[1] = __dadd_rn(__dadd_rn(o[1], __dadd_rn(__dmul_rn(o[5], xl[0]), __dmul_rn(o[6], xl[1]))),
                     __dadd_rn(__dmul_rn(o[10], xr[0]), __dmul_rn(o[11], xr[1])));
    x[2] = __dadd_rn(__dadd_rn(o[2], __dmul_rn(o[7], xl[2])), __dmul_rn(o[12], xr[2]));
}

}  // namespace holo
}  // namespace keq
