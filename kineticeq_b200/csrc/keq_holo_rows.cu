// keq_holo_rows.cu -- the HOLO step with one CTA per row block, for instances
// whose blocks are all resident (several instances share a launch while their
// blocks fit the chip).  Same method and phases as keq_holo.cu, which has the
// reference lines; the work is cut and synchronised like keq_implicit_solo.cu:
//
//  - a CTA owns up to 32 rows of one instance with all velocities: the explicit
//    term, the Maxwellian sums, the distribution sweep (keq_rows.cuh) and the
//    row moments need no other CTA except through the sweep's block maps;
//  - the first lo_n CTAs of an instance also own a chunk of up to 32 rows of
//    the low-order (LO) system, solved by one warp: by sweeps over a window
//    (lo_solve) or, beyond their bound, by cyclic reduction (lo_general);
//  - CTAs meet through tagged words (TaggedMaps): row moments to the LO chunks,
//    LO interface data and residuals between the chunks, LO solutions back to
//    the blocks, HO residuals between the blocks.  There is one grid barrier,
//    behind the prologue.
//
// LO iteration.  A chunk's warp works on a window of its rows and 16 on either
// side (two rows per lane).  With q = 2 c |u|, c = dt/(4 dx), the rows of the LO
// system are x = D - N x with ||N|| <= q / (1 - q) in the norm that weighs nu by
// 1/max(|u|, 1/2), so red-black Gauss-Seidel sweeps from the previous iterate
// reach its solution to 2^-60 in at most 8 sweeps, and what lies 16 rows away
// contributes less than that, while q / (1 - q) <= 2^(-30/8) = 0.0743 (CFL 0.9
// and v_max = 10: |u| <= 1.5).  One warp sweeps the window, two read the new rows
// of the neighbouring chunks, which the next iteration needs, and one the
// residuals of all chunks, which it does not: the decision on an iteration is
// taken behind the work of the next (lo_solve).  A chunk that does not meet the
// bound raises a flag in its residual; from that iteration on the HO iteration's
// LO systems are solved by warp-parallel PCR with explicit interface unknowns,
// x = y + P xi_{k-1} + Q xi_k (lo_general).
//
// What bounds it: the latency of the LO chain.  With grid barriers, a single CTA
// solving the interfaces and IEEE divisions in the PCR an LO iteration of
// 4096x512 took 29 us on one B200, with the rest of the chip waiting; PCR chunks
// with one exchange took 23 us (a warp alone spends about 10 cycles an
// instruction, and the polling warps of its CTA took issue slots from it).  With
// the windows an iteration takes 3 us, 2.3 since none waits for all residuals.
// us per step: 4096x512 2620 with the look-back kernel, 1626 PCR chunks, 429
// (kernel alone) windows, 383 decision one iteration behind, 366 preparation per
// cell; 256x128 508, 304, 115.5, 109.6, 103.9.  The LO iterations are about half
// of that, the sweep a quarter.
#include <cuda_runtime.h>

#include "keq_holo.cuh"
#include "keq_rows.cuh"

namespace keq {
namespace holo {

using rows::kBadValue;
using rows::kBadWait;
using rows::kRows;
using rows::ld_tagged;
using rows::st_tagged;
using rows::Tile;
using rows::TileBuf;

constexpr int kMaxWarps = 16;
constexpr int kSignSlots = 8;  // partial-sum slots per sign of v
constexpr int kHalo = 16, kWin = 64;  // LO window: rows on either side, rows
// Largest q0 = 2 c max(|u|, 1/2) that N = 1 .. 8 window sweeps suffice for:
// q0 / (1 - q0) <= 2^(-30/N), a little less.
__constant__ double kLoQ[8] = {9.313225728168e-10, 3.051664680033e-05, 0.000975609755122, 0.005493921805589, 0.01538461536923, 0.03030303027273, 0.04877045182659, 0.06918336057372};
constexpr int kLoRec = 40;   // 16-byte units of an LO record (33 used)
constexpr int kRecFirst = 0, kRecLast = 13, kRecAl = 26, kRecStd = 31, kRecDf = 32, kRecUsed = 33;

struct alignas(16) HoloSmem : rows::BlockSmemT<HoloInst> {
    double R[kRows][8];        // raw half-range sums of f_z (the block's rows)
    double Ms[kRows][3];       // velocity sums of M(f_z)
    double Wl[kRows][3];       // LO solution of the block's rows
    double cmax[kMaxWarps];    // largest Maxwellian coefficient over the LO chunks, per warp
    double Rb[2][8];           // raw sums of the boundary rows
    double red[kMaxWarps][3];
    double all[2][kMaxWarps][4];  // per warp: HO residuals over the blocks read, by parity
    // LO chunk
    double row[kWin + 2][12];   // raw sums and Maxwellian sums of the window's rows and their neighbours
    double cell[kWin + 2][7];   // Q, fluxes, collision term of those cells (lo_cell)
    double prep[kWin][6];       // T1, Y of the window's rows
    double win[kWin][3];        // LO iterate of the window's rows
    double halo[2][2 * kHalo][3];  // neighbours' new rows, by parity
    double lres[2];             // residual maximum of the chunks, or a flag (< 0), by parity
    double lmy[2];              // largest |Y| of the window's halves
    double out[kRecUsed];       // record
    double gen[2][2];           // general solve, by parity: residual maximum, flag over the chunks
    double nbr[2][2][13];       // by parity: next chunk's first row, previous chunk's last row
    double xi[3][3];            // interface values k-1, k, k+1 (general solve)
    double lo_std;
    int lo_state[2];            // outcome of the windows (kLo...), iterations
    unsigned lo_seq[2];         // exchanges so far, exchange of the solution
    int lo_fail;                // a wait gave up
    int bad[2];                 // flags of the sweep (kBad...), by parity
    int set;                    // launch parity
};

// Moments and Maxwellian coefficients with the short division and root.
__device__ __forceinline__ Mom mom_nr(const double* R8, double dv) {
    Mom m;
    m.n = (R8[0] + R8[4]) * dv;
    m.s1 = (R8[1] + R8[5]) * dv;
    m.s2 = (R8[2] + R8[6]) * dv;
    m.s3 = (R8[3] + R8[7]) * dv;
    m.u = div_nr(m.s1, m.n);
    m.T = div_nr(m.s2, m.n) - m.u * m.u;
    return m;
}
__device__ __forceinline__ void mc_nr(double n, double u, double T, double tau_tilde, double* c4) {
    double sT, y;
    sqrt_nr(T, sT, y);
    const double a = n * kInvSqrt2Pi;
    c4[0] = u;
    c4[1] = -div_nr(0.5, T);
    c4[2] = refined(a * y, sT, a, y);
    c4[2] = rows::amplitude(c4);
    c4[3] = div_nr(n * sT, tau_tilde);
}

// Partial-sum slot of a v-tile: each sign of v has its own set of nslot.  A slot
// is one warp's (with 16 warps a sign has at most 8 tiles).
__device__ __forceinline__ int slot_of(const HoloInst& I, int nslot, int vt, bool& first) {
    const int t = vt >= I.nt_neg ? vt - I.nt_neg : vt;
    first = t < kSignSlots;
    return (vt >= I.nt_neg ? nslot : 0) + (t & (kSignSlots - 1));
}
// Raw half-range sum q (0-3: v > 0; 4-7: v <= 0) of the lane's row.
__device__ __forceinline__ double half_sum(const HoloInst& I, const double (*part)[4][32], int nslot, int q) {
    return q < 4 ? rows::slot_sum<4, kSignSlots>(part + nslot, I.nvt - I.nt_neg, q)
                 : rows::slot_sum<4, kSignSlots>(part, I.nt_neg, q - 4);
}

// Sums over the velocities of a Maxwellian times (1, v, v^2/2), one warp, four
// velocities per lane in flight.
__device__ __forceinline__ void maxwell_sums4(const double* v, int nv, const double* c4, double* s3) {
    const int lane = threadIdx.x & 31;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    for (int j0 = lane; j0 < nv; j0 += 128) {
        double x[4], M[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) x[t] = __ldg(&v[j0 + 32 * t < nv ? j0 + 32 * t : j0]);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const double d = x[t] - c4[0];
            M[t] = c4[2] * rows::exp_neg(d * d * c4[1]);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const double Mt = j0 + 32 * t < nv ? M[t] : 0.0;
            a0 += Mt;
            a1 = fma(Mt, x[t], a1);
            a2 = fma(Mt * x[t], x[t], a2);
        }
    }
    s3[0] = warp_sum(a0);
    s3[1] = warp_sum(a1);
    s3[2] = 0.5 * warp_sum(a2);
}

// A boundary row (one warp): raw sums, W_HO, the constant consistency term and
// its Maxwellian sums, its copy into f_out.
__device__ __noinline__ void boundary_row_h(const HoloInst& I, const double* fn, double* fo, int side,
                                            double* misc) {
    const int lane = threadIdx.x & 31;
    const size_t ib = side == 0 ? 0 : (size_t)(I.nx - 1);
    double R8[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    double mx = 0.0;
    for (int j = lane; j < I.nv; j += 32) {
        const double x = __ldcg(&fn[ib * I.nv + j]), v = __ldg(&I.v[j]);
        fo[ib * I.nv + j] = x;
        const double t1 = x * v, t2 = t1 * v, t3 = t2 * v;
        const bool pos = v > 0.0;
        R8[0] += pos ? x : 0.0;
        R8[1] += pos ? t1 : 0.0;
        R8[2] += pos ? t2 : 0.0;
        R8[3] += pos ? t3 : 0.0;
        R8[4] += pos ? 0.0 : x;
        R8[5] += pos ? 0.0 : t1;
        R8[6] += pos ? 0.0 : t2;
        R8[7] += pos ? 0.0 : t3;
        mx = nan_max(mx, fabs(x));
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) R8[q] = warp_sum(R8[q]);
    mx = warp_max(mx);
    const Mom m = mom_of(R8, I.dv);
    double c4[4], sm[3];
    mc_of(m, I.tau_tilde, c4);
    maxwell_sums_row(I.v, I.nv, c4, sm);
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 8; ++q) I.Rn[8 * ib + q] = R8[q];
        I.Who[3 * ib + 0] = m.n;
        I.Who[3 * ib + 1] = m.n * m.u;
        I.Who[3 * ib + 2] = 0.5 * m.n * (m.u * m.u + m.T);
        const double sfw[3] = {m.n, m.s1, 0.5 * m.s2};
        double my = 0.0;
        for (int q = 0; q < 3; ++q)
            my = nan_max(my, fabs(I.con_terms ? I.dt * (((sm[q] * I.dv) - sfw[q]) * c4[3]) : 0.0));
        atomic_max_nonneg(&misc[0], mx);
        atomic_max_nonneg(&misc[1], my);
        const double den = m.n + 1e-30;
        const double u = (m.n * m.u) / den;
        double T = 2.0 * ((0.5 * m.n * (m.u * m.u + m.T)) / den - 0.5 * u * u);
        T = (T != T || T >= 1e-30) ? T : 1e-30;
        I.Wlo[ib] = m.n;
        I.Wlo[I.nx + ib] = u;
        I.Wlo[2 * (size_t)I.nx + ib] = T;
    }
}

// Explicit term of one tile (f^n is in w.a) into HBM; the tile buffer is left
// with the Maxwellian of f^n.  C.coef holds u, -1/(2T), n/sqrt(2 pi T), 1/tau
// in both scan orders.  Returns the lane's largest |E|.
__device__ __forceinline__ double explicit_tile_h(const HoloSmem& C, TileBuf& w, const Tile& g,
                                                  const double* __restrict__ fn) {
    const HoloInst& I = C.I;
    const int lane = threadIdx.x & 31;
    double prev = __ldcg(fn + g.first - g.st);
    cp_async_wait_all();
    const double vj = w.vw[lane].x;
    w.vw[lane].y = vj * vj;
    const double(*co)[4] = C.coef[g.pos ? 0 : 1];
    const double vc = (-vj) / I.dx;
    const double a = (1.0 - kTheta) * I.dt;
    double* e_out = I.E + g.first;
    double mx = 0.0;
#pragma unroll 4
    for (int r = 0; r < g.nr; ++r) {
        const double f = w.a[r][lane];
        const double d = vj - co[r][0];
        const double M = co[r][2] * rows::exp_neg(d * d * co[r][1]);
        // bgk1d_compute_streaming.py: (f_i - f_{i-1}) (-v/dx) for v > 0,
        // (f_{i+1} - f_i) (-v/dx) for v <= 0
        const double st = g.pos ? (f - prev) * vc : (prev - f) * vc;
        const double col = (M - f) * co[r][3];
        const double e = f + a * (st + col);
        if (g.lane_ok) e_out[(long long)r * g.st] = e;
        mx = fabs(e) > mx ? fabs(e) : mx;
        prev = f;
        w.a[r][lane] = M;
    }
    __syncwarp();
    return mx;
}

// Residuals of the HO iteration: |x - o| / (abs_tol + tol ref), max |x - o|,
// max ref.
struct HoResidual {
    FracMax q1;
    double mdf, mref, tol, abs_tol;
    bool strict;
    __device__ __forceinline__ HoResidual(double t, double a)
        : mdf(0.0), mref(0.0), tol(t), abs_tol(a), strict(!(a > 1e-290 && t >= 0.0)) {}
    __device__ __forceinline__ void add(double x, double o) {
        const double df = fabs(x - o);
        const double ref = fabs(x) > fabs(o) ? fabs(x) : fabs(o);
        const double b1 = fma(tol, ref, abs_tol);
        if (strict) {
            q1.add(df, b1);
        } else {
            const bool t1 = df * q1.den > q1.num * b1;
            q1.num = t1 ? df : q1.num;
            q1.den = t1 ? b1 : q1.den;
        }
        mdf = df > mdf ? df : mdf;
        mref = ref > mref ? ref : mref;
    }
    __device__ __forceinline__ void add4(const double (&x)[4], const double (&o)[4]) {
        if (strict) {
#pragma unroll
            for (int t = 0; t < 4; ++t) add(x[t], o[t]);
            return;
        }
        double n[4], d[4], m[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            m[t] = fabs(x[t]) > fabs(o[t]) ? fabs(x[t]) : fabs(o[t]);
            n[t] = fabs(x[t] - o[t]);
            d[t] = fma(tol, m[t], abs_tol);
        }
        const double a = n[0] > n[1] ? n[0] : n[1], b = n[2] > n[3] ? n[2] : n[3];
        const double c = m[0] > m[1] ? m[0] : m[1], e = m[2] > m[3] ? m[2] : m[3];
        mdf = a > mdf ? a : mdf;
        mref = c > mref ? c : mref;
        mdf = b > mdf ? b : mdf;
        mref = e > mref ? e : mref;
        rows::larger(n[0], d[0], n[1], d[1]);
        rows::larger(n[2], d[2], n[3], d[3]);
        rows::larger(n[0], d[0], n[2], d[2]);
        rows::larger(q1.num, q1.den, n[0], d[0]);
    }
    __device__ __forceinline__ void set_nan() {
        q1.special = mdf = mref = __longlong_as_double(0x7ff8000000000000ll);
    }
};

// What the LO right-hand sides need of a cell whose sums are row a of C.row:
// C.cell[a] = Q, the momentum-form fluxes F, and (interior cells) the
// consistency term of the collisions.
__device__ __forceinline__ void lo_cell(HoloSmem& C, int a, int i) {
    const HoloInst& I = C.I;
    const Mom m = mom_nr(C.row[a], I.dv);
    const double Q = q_of(m);
    double* o = C.cell[a];
    o[0] = Q;
    const double P = m.n * m.T, nu = m.n * m.u, U = 0.5 * m.n * (m.u * m.u + m.T);
    o[1] = nu;
    o[2] = div_nr(nu * nu, m.n + 1e-30) + P;
    o[3] = (U + P) * m.u + Q;
    if (I.con_terms && i >= 1 && i <= I.nx - 2) {
        double sT, inv;
        sqrt_nr(m.T, sT, inv);
        const double inv_tau_new = div_nr(m.n * sT, I.tau_tilde);
        const double sfw[3] = {m.n, m.s1, 0.5 * m.s2};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double smw = C.row[a][8 + c] * I.dv;
            o[4 + c] = kTheta * ((smw - sfw[c]) * inv_tau_new) + __ldcg(&I.Iold[3 * (size_t)i + c]);
        }
    }
}

// Constant part T1 of the LO right-hand side and the consistency terms Y of
// interior row k (lane; its cells i-1, i, i+1 are a, a+1, a+2 of C.row and
// C.cell) for an HO iteration: lo_prep_row of keq_holo.cu.  Returns max |Y|.
__device__ __forceinline__ double lo_prep(const HoloSmem& C, int k, int a, double* T1, double* Y) {
    const HoloInst& I = C.I;
    const int i = k + 1;
    const double dv = I.dv, dt = I.dt, c2 = I.dtdx2;
    double S[2][3];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        double Lr[4], Rg[4];  // v > 0 sums of the left cell, v <= 0 sums of the right cell
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            Lr[q] = I.con_terms ? C.row[a + s][q] : __ldcg(&I.Rn[8 * (size_t)(i - 1 + s) + q]);
            Rg[q] = I.con_terms ? C.row[a + s + 1][4 + q] : __ldcg(&I.Rn[8 * (size_t)(i + s) + 4 + q]);
        }
        const int o = I.sv_down ? 0 : 1;
        S[s][0] = (Lr[o] + Rg[o]) * dv;
        S[s][1] = (Lr[o + 1] + Rg[o + 1]) * dv;
        S[s][2] = 0.5 * ((Lr[o + 2] + Rg[o + 2]) * dv);
    }
    const double *c0 = C.cell[a], *c1 = C.cell[a + 1], *c2l = C.cell[a + 2];
    double y[3] = {0.0, 0.0, 0.0};
    if (I.con_terms) {
        if (I.flux_cons) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double g0 = -S[0][c] + 0.5 * (c0[1 + c] + c1[1 + c]);
                const double g1 = -S[1][c] + 0.5 * (c1[1 + c] + c2l[1 + c]);
                y[c] = dt * div_nr(g1 - g0, I.dx);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) y[c] = y[c] + dt * c1[4 + c];
    }
    const double QhL = 0.5 * (c0[0] + c1[0]), QhR = 0.5 * (c1[0] + c2l[0]);
    const double Fd[3] = {S[1][0] - S[0][0], S[1][1] - S[0][1],
                          (S[1][2] + 2.0 * QhR) - (S[0][2] + 2.0 * QhL)};
    double mx = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        T1[c] = __dadd_rn(__ldcg(&I.Who[3 * (size_t)i + c]), __dmul_rn(-c2, Fd[c]));
        Y[c] = y[c];
        mx = nan_max(mx, fabs(y[c]));
    }
    return mx;
}

// Largest Maxwellian coefficient that the distribution sweep will use for a row
// of the LO iterate (n, nu, U), up to rounding.
__device__ __forceinline__ void lo_state(const double* W, double& u, double& T) {
    const double den = W[0] + 1e-30;
    u = div_nr(W[1], den);
    T = 2.0 * (div_nr(W[2], den) - 0.5 * u * u);
    T = (T != T || T >= 1e-30) ? T : 1e-30;
}

__device__ __forceinline__ double norm2(const double* M) {  // inf-norm of a 2x2 block
    return fmax(fabs(M[0]) + fabs(M[1]), fabs(M[2]) + fabs(M[3]));
}

// The LO Picard iteration of one HO iteration, by the CTA that owns chunk c
// (all threads).  seq: exchanges so far (the tag, equal in all chunks).
struct LoResult {
    int iters;
    unsigned seq;
    double df, std_res, max_y;
};

// From iteration m0 on with explicit interface unknowns (warp 0 does the rows);
// the iterate is in C.win.  Returns false if a wait gave up.
__device__ __noinline__ bool lo_general(HoloSmem& C, unsigned char* scratch, int c, int z, int m0,
                                        unsigned& seq, unsigned long long limit, LoResult& out) {
    const HoloInst& I = C.I;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int K = I.lo_n;
    const int s = (int)((long long)c * I.n_inner / K);
    const int e = (int)((long long)(c + 1) * I.n_inner / K) - 1;
    const int len = e - s + 1, nloc = len - 1;
    bool ok = true;
    double x[3] = {0.0, 0.0, 0.0}, T1[3], Y[3], wl[3] = {0.0, 0.0, 0.0}, wr[3] = {0.0, 0.0, 0.0};
    double mdf = 0.0, std_prev = 0.0;
    const bool mine = warp == 0 && lane < len;
    if (mine) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            T1[q] = C.prep[kHalo + lane][q];
            Y[q] = C.prep[kHalo + lane][3 + q];
            wl[q] = C.win[kHalo + lane - 1][q];
            x[q] = C.win[kHalo + lane][q];
            wr[q] = C.win[kHalo + lane + 1][q];
        }
    }
    for (int m = m0;; ++m) {
        ++seq;
        ulonglong2* recs = I.lorec + (size_t)(seq & 1u) * K * kLoRec;
        double o[13];
        if (warp == 0) {
            // system m from the iterate in x
            LoRow L{};
            bool flag = false;
            if (mine) {
                lo_row_w<true>(I, s + lane, wl, x, wr, T1, Y, L);
                // near the identity: no pivot of any reduction is small
                const double E4[4] = {L.B[0] - 1.0, L.B[1], L.B[2], L.B[3] - 1.0};
                flag = !(norm2(L.A) + norm2(L.C) + norm2(E4) <= 0.5 &&
                         fabs(L.a) + fabs(L.c) + fabs(L.b - 1.0) <= 0.5);
            }
            PcrRow q;
            local_rows(q, L.A, L.B, L.C, L.D, L.a, L.b, L.c, L.d, lane, nloc);
            warp_pcr(q, nloc);
            if (lane < nloc) {
                rep_of(q, o);
            } else {
#pragma unroll
                for (int t = 0; t < 13; ++t) o[t] = 0.0;
                o[8] = o[11] = o[12] = 1.0;
            }
            // the row before the interface, at the interface's lane
            double pm[13];
#pragma unroll
            for (int t = 0; t < 13; ++t) pm[t] = __shfl_up_sync(0xffffffffu, o[t], 1);
            if (nloc == 0) {
#pragma unroll
                for (int t = 0; t < 13; ++t) pm[t] = 0.0;
                pm[3] = pm[6] = pm[7] = 1.0;
            }
            if (lane == 0) {
#pragma unroll
                for (int t = 0; t < 13; ++t) C.out[kRecFirst + t] = o[t];
                // the first row's dependence on the chunk's own interface
                if (K > 1 && c > 0)
                    flag |= !(norm2(o + 8) <= 8.5e-22 && fabs(o[12]) <= 8.5e-22);  // 2^-70
            }
            if (lane == nloc) {
                double al[4], T4[4], t2[2];
                mm2(L.A, pm + 3, al);
                mm2(L.A, pm + 8, T4);
                mv2(L.A, pm, t2);
                double* r = C.out + kRecLast;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    r[t] = L.B[t] + T4[t];
                    r[8 + t] = L.C[t];
                    C.out[kRecAl + t] = al[t];
                }
                r[4] = fma(L.a, pm[12], L.b);
                r[5] = L.D[0] - t2[0];
                r[6] = L.D[1] - t2[1];
                r[7] = fma(-L.a, pm[2], L.d);
                r[12] = L.c;
                const double as = L.a * pm[7];
                C.out[kRecAl + 4] = as;
                // the interface's dependence on the previous interface
                if (K > 1 && c > 0) flag |= !(norm2(al) <= 5.4e-20 && fabs(as) <= 5.4e-20);  // 2^-64
            }
            flag = __any_sync(0xffffffffu, flag) && K > 1;
            if (lane == 0) {
                // the flag in the sign bit
                C.out[kRecStd] = __hiloint2double(__double2hiint(std_prev) | (flag ? 0x80000000 : 0),
                                                  __double2loint(std_prev));
                C.out[kRecDf] = mdf;
            }
            __syncwarp();
            for (int t = lane; t < kRecUsed; t += 32) st_tagged(recs + (size_t)c * kLoRec + t, C.out[t], seq);
        }
        // All chunks' residuals by one warp, the neighbours' data by another.  One
        // word per chunk and a pause between polls: with all warps of all chunks
        // reading five words each the iteration took 170 us at 5806x194.
        if (warp == 1) {
            double a = 0.0;
            bool fl = false;
            for (int j = lane; j < K; j += 32) {
                const ulonglong2* p = recs + (size_t)j * kLoRec + kRecStd;
                double y;
                unsigned long long it = 0;
                while (!ld_tagged(p, seq, y)) {
                    if (++it > limit) {
                        ok = false;
                        break;
                    }
                    if (it < 1000000ull) __nanosleep(200);
                }
                fl |= __double2hiint(y) < 0;
                a = __double_as_longlong(fabs(y)) > __double_as_longlong(a) ? fabs(y) : a;
            }
            __syncwarp();
            fl = __any_sync(0xffffffffu, fl);
            a = rows::warp_max_bits(a);
            if (lane == 0) {
                C.gen[seq & 1u][0] = a;
                C.gen[seq & 1u][1] = fl ? 1.0 : 0.0;
            }
        } else if (warp == 2 && lane < 26) {
            const bool nxt = lane < 13;
            const int q = nxt ? lane : lane - 13;
            const int oc = nxt ? c + 1 : c - 1;
            double a = 0.0;
            if (oc >= 0 && oc < K) {
                unsigned long long it = 0;
                while (!ld_tagged(recs + (size_t)oc * kLoRec + (nxt ? kRecFirst : kRecLast) + q, seq, a)) {
                    if (++it > limit) {
                        ok = false;
                        break;
                    }
                    if (it < 1000000ull) __nanosleep(100);
                }
            }
            C.nbr[seq & 1u][nxt ? 0 : 1][q] = a;
        }
        if (!__syncthreads_and(ok)) return false;
        const double res = C.gen[seq & 1u][0];
        const bool coupled = C.gen[seq & 1u][1] != 0.0;
        out.iters = m;
        out.std_res = res;
        out.df = -2.0;  // in the records of exchange out.seq
        out.seq = seq;
        // (a step of this loop has been done before there is a residual)
        const bool conv = m > m0 && (I.fixed_lo > 0 ? m >= I.fixed_lo : res < 1.0);
        if (conv || m >= I.lo_iter) {
            if (mine) {
                ulonglong2* wp = I.wlo + 4 * (size_t)(s + lane + 1);
#pragma unroll
                for (int q = 0; q < 3; ++q) st_tagged(wp + q, x[q], (unsigned)z + 1u);
            }
            if (warp == 0) {
                double cm = 0.0;
                if (mine) {
                    double u, T, r, y;
                    lo_state(x, u, T);
                    sqrt_nr(T, r, y);
                    cm = fabs(x[0] * kInvSqrt2Pi * y);
                }
                cm = rows::warp_max_bits(cm);
                if (lane == 0) st_tagged(I.locm + c, cm, (unsigned)z + 1u);
            }
            return true;
        }
        double xl[3], xr[3];  // interface values of the previous chunk and of this one
        double wn0[3];        // next chunk's first row
        if (!coupled) {
            if (warp == 0) {
                // both from one formula: xi = (last part + C first row)^-1 (...)
                auto iface = [&](const double* last, const double* first, bool coupled, double* xo) {
                    double be[4], de[2], bs = last[4], ds = last[7];
#pragma unroll
                    for (int t = 0; t < 4; ++t) be[t] = last[t];
                    de[0] = last[5];
                    de[1] = last[6];
                    if (coupled) {
                        double U4[4], u2[2];
                        mm2(last + 8, first + 3, U4);
                        mv2(last + 8, first, u2);
#pragma unroll
                        for (int t = 0; t < 4; ++t) be[t] += U4[t];
                        de[0] -= u2[0];
                        de[1] -= u2[1];
                        bs = fma(last[12], first[7], bs);
                        ds = fma(-last[12], first[2], ds);
                    }
                    double Bi[4];
                    inv2(be, Bi);
                    mv2(Bi, de, xo);
                    xo[2] = ds * rcp_or0(bs);
                };
                iface(C.out + kRecLast, C.nbr[seq & 1u][0], c + 1 < K, xr);
                if (c > 0)
                    iface(C.nbr[seq & 1u][1], C.out + kRecFirst, true, xl);
                else
                    xl[0] = xl[1] = xl[2] = 0.0;
                const double zero[3] = {0.0, 0.0, 0.0};
                rep_apply(C.nbr[seq & 1u][0], xr, zero, wn0);
            }
        } else {
            // general: the whole interface system from all records
            lo_reduced_solve(
                K, scratch,
                [&](int k, double* al, double* be, double* ga, double* de, double* s4) {
                    double r[18], f[13];
                    // the 31 words together
                    const ulonglong2* p = recs + (size_t)k * kLoRec + kRecLast;
                    const ulonglong2* p1 = recs + (size_t)(k + 1 < K ? k + 1 : k) * kLoRec + kRecFirst;
                    unsigned long long it = 0;
                    for (;;) {
                        bool there = true;
#pragma unroll
                        for (int t = 0; t < 18; ++t) there &= ld_tagged(p + t, seq, r[t]);
#pragma unroll
                        for (int t = 0; t < 13; ++t) there &= ld_tagged(p1 + t, seq, f[t]);
                        if (there) break;
                        if (++it > limit) {
                            *(volatile int*)&C.lo_fail = 1;
                            break;
                        }
                        __nanosleep(100);
                    }
#pragma unroll
                    for (int t = 0; t < 13; ++t) f[t] = k + 1 < K ? f[t] : 0.0;
                    double U4[4], u2[2];
                    mm2(r + 8, f + 3, U4);
                    mm2(r + 8, f + 8, ga);
                    mv2(r + 8, f, u2);
                    for (int t = 0; t < 4; ++t) {
                        be[t] = r[t] + U4[t];
                        al[t] = k > 0 ? r[13 + t] : 0.0;
                    }
                    de[0] = r[5] - u2[0];
                    de[1] = r[6] - u2[1];
                    s4[0] = k > 0 ? r[17] : 0.0;
                    s4[1] = fma(r[12], f[7], r[4]);
                    s4[2] = r[12] * f[12];
                    s4[3] = fma(-r[12], f[2], r[7]);
                },
                [&](int k, double x0, double x1, double x2) {
                    const int q = k - c + 1;
                    if (q >= 0 && q < 3) {
                        C.xi[q][0] = x0;
                        C.xi[q][1] = x1;
                        C.xi[q][2] = x2;
                    }
                });
            __syncthreads();
            if (*(volatile int*)&C.lo_fail) return false;
            if (warp == 0) {
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    xl[q] = c > 0 ? C.xi[0][q] : 0.0;
                    xr[q] = C.xi[1][q];
                }
                const double x2[3] = {c + 1 < K ? C.xi[2][0] : 0.0, c + 1 < K ? C.xi[2][1] : 0.0,
                                      c + 1 < K ? C.xi[2][2] : 0.0};
                rep_apply(C.nbr[seq & 1u][0], xr, x2, wn0);
            }
        }
        if (warp == 0) {
            // recovery, residual, neighbours of the next system
            double df1 = 0.0;
            FracMax fm;
            if (mine) {
                double xn[3];
                rep_apply(o, xl, xr, xn);
                if (lane == nloc) {
                    xn[0] = xr[0];
                    xn[1] = xr[1];
                    xn[2] = xr[2];
                }
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const double df = fabs(xn[q] - x[q]);
                    const double ref = nan_max(fabs(xn[q]), fabs(x[q]));
                    df1 = nan_max(df1, df);
                    fm.add(df, I.lo_abs_tol + I.lo_tol * ref);
                    x[q] = xn[q];
                }
            }
            const double fv = fm.special != fm.special || fm.special > 0.0 ? fm.value() : div_nr(fm.num, fm.den);
            mdf = rows::warp_max_bits(df1);
            std_prev = rows::warp_max_bits(fv);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                wl[q] = __shfl_up_sync(0xffffffffu, x[q], 1);
                wr[q] = __shfl_down_sync(0xffffffffu, x[q], 1);
            }
            if (lane == 0)
#pragma unroll
                for (int q = 0; q < 3; ++q) wl[q] = c > 0 ? xl[q] : __ldcg(&I.Who[q]);
            if (lane == nloc)
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    wr[q] = c + 1 < K ? wn0[q] : __ldcg(&I.Who[3 * (size_t)(I.nx - 1) + q]);
        }
    }
}

// Named barriers of the first four warps: rows of the neighbours are there
// (warps 0-2), residuals of the chunks are there (warps 0 and 3), decision
// (warp 0 arrives, the others wait).
__device__ __forceinline__ void bar_rows() { asm volatile("bar.sync 1, 96;" ::: "memory"); }
__device__ __forceinline__ void bar_res() { asm volatile("bar.sync 2, 64;" ::: "memory"); }
__device__ __forceinline__ void bar_tell() { asm volatile("bar.arrive 3, 128;" ::: "memory"); }
__device__ __forceinline__ void bar_told() { asm volatile("bar.sync 3, 128;" ::: "memory"); }
constexpr int kLoDone = 0, kLoGeneral = 1, kLoFailed = 2, kLoGoOn = 3;

// The LO Picard iteration by windows (see the head of the file).
__device__ __noinline__ bool lo_solve(HoloSmem& C, unsigned char* scratch, int c, int z, unsigned& seq,
                                      unsigned long long limit, LoResult& out) {
    const HoloInst& I = C.I;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int K = I.lo_n, n = I.n_inner;
    const int s = (int)((long long)c * n / K);
    const int e = (int)((long long)(c + 1) * n / K) - 1;
    const int w0 = s - kHalo;  // interior row of window position 0
    bool ok = true;
    // raw sums of the cells of interior rows w0-1 .. w0+64 that exist
    // (six words per thread in flight: with four warps one after another took 5000
    // cycles)
    for (int t0 = tid; t0 < (kWin + 2) * 11; t0 += 6 * blockDim.x) {
        double v[6];
        const ulonglong2* p[6];
        bool want[6];
#pragma unroll
        for (int h = 0; h < 6; ++h) {
            const int t = t0 + h * (int)blockDim.x;
            const int rr = t / 11, q = t - 11 * rr, i = w0 + rr;  // cell
            const bool used = t < (kWin + 2) * 11 && i >= 0 && i < I.nx && i <= e + kHalo + 2;
            const bool edge = i == 0 || i == I.nx - 1;
            want[h] = used && !edge;
            p[h] = I.rowd + (want[h] ? 12 * (size_t)i + q : 12);
            v[h] = used && edge ? (q < 8 ? C.Rb[i == 0 ? 0 : 1][q] : 0.0) : 1.0;
        }
        unsigned long long it = 0;
        for (;;) {
            bool there = true;
#pragma unroll
            for (int h = 0; h < 6; ++h)
                if (want[h]) there &= ld_tagged(p[h], (unsigned)z + 1u, v[h]);
            if (there) break;
            if (++it > limit) {
                ok = false;
                break;
            }
        }
#pragma unroll
        for (int h = 0; h < 6; ++h) {
            const int t = t0 + h * (int)blockDim.x;
            if (t < (kWin + 2) * 11) C.row[t / 11][t % 11] = v[h];
        }
    }
    __syncthreads();
    if (tid < kWin + 2) lo_cell(C, tid, w0 + tid);
    __syncthreads();
    // T1, Y and W_HO of the window's rows
    double my = 0.0;
    if (tid < kWin) {
        const int k = w0 + tid, i = k + 1;
        const int ic = i < 0 ? 0 : (i > I.nx - 1 ? I.nx - 1 : i);
        double T1[3] = {0.0, 0.0, 0.0}, Y[3] = {0.0, 0.0, 0.0};
        if (k >= 0 && k < n && k <= e + kHalo) {
            const double y = lo_prep(C, k, tid, T1, Y);
            if (k >= s && k <= e) my = y;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            C.prep[tid][q] = T1[q];
            C.prep[tid][3 + q] = Y[q];
            C.win[tid][q] = __ldcg(&I.Who[3 * (size_t)ic + q]);
        }
        my = warp_max(my);
        if (lane == 0) C.lmy[warp] = my;
    }
    if (!__syncthreads_and(ok)) return false;
    my = nan_max(C.lmy[0], C.lmy[1]);
    if (c == 0) my = nan_max(my, __ldcg(&I.misc[4 * C.set + 1]));
    const double c4 = 0.5 * I.dtdx2, c2 = I.dtdx2;
    double x[2][3], D0[2], T1a[2], Ya[2], T1b[2], Yb[2];
    bool in[2], own[2];
    int hid[2];  // the row's place among the neighbours' rows
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int p = 2 * lane + h, k = w0 + p;
        in[h] = k >= 0 && k < n && k <= e + kHalo;  // the others stay as they are
        own[h] = k >= s && k <= e;
        hid[h] = !in[h] || own[h] ? 0 : (k < s ? p : kHalo + k - e - 1);
#pragma unroll
        for (int q = 0; q < 3; ++q) x[h][q] = C.win[p][q];
        D0[h] = __dadd_rn(C.prep[p][0], C.prep[p][3]);
        T1a[h] = C.prep[p][1];
        Ya[h] = C.prep[p][4];
        T1b[h] = C.prep[p][2];
        Yb[h] = C.prep[p][5];
    }
    // iteration i of warp 0: rows and residual out; the decision on iteration
    // i-1, whose residuals had an iteration's time to arrive; neighbours' rows in
    const int most = I.fixed_lo > 0 && I.fixed_lo < I.lo_iter ? I.fixed_lo : I.lo_iter;
    const unsigned seq0 = seq + 1;  // exchange of iteration 0
    if (warp == 0) {
        double xp[2][3];  // the iterate before x
        int state = kLoGoOn;
        double all = 0.0;
        for (int i = 0;; ++i) {
            const unsigned sq = seq0 + i, par = sq & 1u;
            double xn[2][3], mdf = 0.0, std_res = 0.0;
            if (i < most) {
                ulonglong2* wx = I.lowx + (size_t)par * 3 * n;
                ulonglong2* lr = I.lores + (size_t)(sq & 3u) * K * 2;
                // u*, P* of the cells (star_of)
                double us[2], Ps[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double den = x[h][0] + 1e-30;
                    us[h] = div_nr(x[h][1], den);
                    double Ts = 2.0 * (div_nr(x[h][2], den) - 0.5 * us[h] * us[h]);
                    Ts = (Ts != Ts || Ts >= 1e-30) ? Ts : 1e-30;
                    Ps[h] = x[h][0] * Ts;
                }
                // half values at the faces left of row a, between a and b, right of b
                const double uP = __shfl_up_sync(0xffffffffu, us[1], 1), PP = __shfl_up_sync(0xffffffffu, Ps[1], 1);
                const double uN = __shfl_down_sync(0xffffffffu, us[0], 1), PN = __shfl_down_sync(0xffffffffu, Ps[0], 1);
                const double uh[3] = {0.5 * (uP + us[0]), 0.5 * (us[0] + us[1]), 0.5 * (us[1] + uN)};
                const double Ph[3] = {0.5 * (PP + Ps[0]), 0.5 * (Ps[0] + Ps[1]), 0.5 * (Ps[1] + PN)};
                double kL[2], kR[2], mL[2], mR[2], b2[2], sL[2], sR[2], bi[2], D1[2], d[2], am = 0.0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = w0 + 2 * lane + h;
                    const double uL = uh[h], uR = uh[h + 1], uL2 = uL * uL, uR2 = uR * uR;
                    // the couplings to the boundary cells and beyond the window are not there
                    kL[h] = k >= 1 && in[h] ? c4 : 0.0;
                    kR[h] = k <= n - 2 && in[h] ? c4 : 0.0;
                    mL[h] = kL[h] * uL2;
                    mR[h] = kR[h] * uR2;
                    sL[h] = kL[h] * uL;
                    sR[h] = kR[h] * uR;
                    b2[h] = (uR2 - uL2) * c4;
                    bi[h] = recip3((uR - uL) * c4 + 1.0);
                    const double bd1 = Ph[h + 1] - Ph[h], bd2 = uR * Ph[h + 1] - uL * Ph[h];
                    D1[h] = __dadd_rn(__dadd_rn(T1a[h], __dmul_rn(-c2, bd1)), Ya[h]);
                    d[h] = __dadd_rn(__dadd_rn(T1b[h], __dmul_rn(-c2, bd2)), Yb[h]);
                    // (lane 0's left and lane 31's right face have no cell behind them)
                    const double ul = lane == 0 && h == 0 ? uR : uL, ur = lane == 31 && h == 1 ? uL : uR;
                    // (by bits: a NaN is above all)
                    const long long ub = __double_as_longlong(fabs(ul)), vb = __double_as_longlong(fabs(ur));
                    const double au = __longlong_as_double(ub > vb ? ub : vb);
                    am = in[h] && __double_as_longlong(au) > __double_as_longlong(am) ? au : am;
                }
                am = rows::warp_max_bits(am);
                // sweeps: q^(2 N) <= 2^-60, q = q0 / (1 - q0)
                const double q0 = 2.0 * c4 * (am <= 0.5 ? 0.5 : am);
                const bool flag = !(q0 <= kLoQ[7]);
                int N = 1;
#pragma unroll
                for (int t = 0; t < 7; ++t) N += q0 > kLoQ[t] ? 1 : 0;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int t = 0; t < 3; ++t) xn[h][t] = x[h][t];
                if (!flag) {
#pragma unroll 1
                    for (int it = 0; it < N; ++it) {
                        // rows a from rows b of this lane and the one before, then the reverse
                        const double nL = __shfl_up_sync(0xffffffffu, xn[1][0], 1),
                                     vL = __shfl_up_sync(0xffffffffu, xn[1][1], 1),
                                     UL = __shfl_up_sync(0xffffffffu, xn[1][2], 1);
                        if (in[0] && lane > 0) {
                            xn[0][0] = fma(-kR[0], xn[1][1], fma(kL[0], vL, D0[0]));
                            xn[0][1] = fma(-b2[0], xn[0][0], fma(-mR[0], xn[1][0], fma(mL[0], nL, D1[0])));
                            xn[0][2] = fma(-sR[0], xn[1][2], fma(sL[0], UL, d[0])) * bi[0];
                        }
                        const double nR = __shfl_down_sync(0xffffffffu, xn[0][0], 1),
                                     vR = __shfl_down_sync(0xffffffffu, xn[0][1], 1),
                                     UR = __shfl_down_sync(0xffffffffu, xn[0][2], 1);
                        if (in[1] && lane < 31) {
                            xn[1][0] = fma(-kR[1], vR, fma(kL[1], xn[0][1], D0[1]));
                            xn[1][1] = fma(-b2[1], xn[1][0], fma(-mR[1], nR, fma(mL[1], xn[0][0], D1[1])));
                            xn[1][2] = fma(-sR[1], UR, fma(sL[1], xn[0][2], d[1])) * bi[1];
                        }
                    }
                }
                // new rows to the neighbours, then the residual to all
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (own[h]) {
                        ulonglong2* p = wx + 3 * (size_t)(w0 + 2 * lane + h);
#pragma unroll
                        for (int t = 0; t < 3; ++t) st_tagged(p + t, xn[h][t], sq);
                    }
                double rn[6], rd[6], dm[6];
                bool odd = false;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int t = 0; t < 3; ++t) {
                        const double df = fabs(xn[h][t] - x[h][t]);
                        const double a = fabs(xn[h][t]), b = fabs(x[h][t]);
                        const double den = I.lo_abs_tol + I.lo_tol * (a > b ? a : b);
                        odd |= own[h] && !(den > 1e-140 && den < 1e140 && df < 1e140);
                        dm[3 * h + t] = rn[3 * h + t] = own[h] ? df : 0.0;
                        rd[3 * h + t] = own[h] ? den : 1.0;
                    }
#pragma unroll
                for (int t = 0; t < 3; ++t) rows::larger(rn[t], rd[t], rn[3 + t], rd[3 + t]);
                rows::larger(rn[0], rd[0], rn[1], rd[1]);
                rows::larger(rn[0], rd[0], rn[2], rd[2]);
                std_res = div_nr(rn[0], rd[0]);
                // (by bits: a NaN is above all)
#pragma unroll
                for (int t = 0; t < 6; ++t)
                    mdf = __double_as_longlong(dm[t]) > __double_as_longlong(mdf) ? dm[t] : mdf;
                if (__any_sync(0xffffffffu, odd)) {  // zero denominators, non-finite values
                    FracMax fm;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int t = 0; t < 3; ++t)
                            if (own[h])
                                fm.add(fabs(xn[h][t] - x[h][t]),
                                       I.lo_abs_tol + I.lo_tol * nan_max(fabs(xn[h][t]), fabs(x[h][t])));
                    std_res = fm.value();
                }
                std_res = rows::warp_max_bits(fabs(std_res));
                if (lane == 0) st_tagged(lr + c, flag ? -1.0 : std_res, sq);
                mdf = rows::warp_max_bits(fabs(mdf));
                if (lane == 0) st_tagged(lr + K + c, mdf, sq);
            }
            if (i > 0) {
                bar_res();
                all = C.lres[(sq - 1u) & 1u];
                if (*(volatile int*)&C.lo_fail) state = kLoFailed;
                else if (all < 0.0) state = kLoGeneral;  // iteration i-1 again, from xp
                else if (i >= most || (I.fixed_lo <= 0 && all < 1.0)) state = kLoDone;
                if (lane == 0) C.lo_state[0] = state;
                __syncwarp();
                bar_tell();
                if (state != kLoGoOn) {
                    if (lane == 0) {
                        C.lo_state[1] = state == kLoGeneral ? i - 1 : i;
                        C.lo_seq[0] = i < most ? sq : sq - 1u;
                        C.lo_seq[1] = sq - 1u;
                        C.lo_std = all;
                    }
                    break;
                }
            }
            bar_rows();
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    const double v = C.halo[par][hid[h]][t];
                    xp[h][t] = x[h][t];
                    x[h][t] = own[h] ? xn[h][t] : (in[h] ? v : x[h][t]);
                }
        }
        if (state == kLoDone) {
            // the solution, and the chunk's largest Maxwellian coefficient
            double cm = 0.0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (own[h]) {
                    ulonglong2* wp = I.wlo + 4 * (size_t)(w0 + 2 * lane + h + 1);
#pragma unroll
                    for (int t = 0; t < 3; ++t) st_tagged(wp + t, x[h][t], (unsigned)z + 1u);
                    double u, T, r, y;
                    lo_state(x[h], u, T);
                    sqrt_nr(T, r, y);
                    const double cc = fabs(x[h][0] * kInvSqrt2Pi * y);
                    cm = !(cc <= cm) ? cc : cm;
                }
            }
            cm = rows::warp_max_bits(cm);
            if (lane == 0) st_tagged(I.locm + c, cm, (unsigned)z + 1u);
        }
        if (state == kLoGeneral) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int t = 0; t < 3; ++t) C.win[2 * lane + h][t] = xp[h][t];
        }
    } else if (warp < 3) {
        // the neighbours' rows next to the chunk: 32 rows, 16 before s, 16 behind e
        for (int i = 0;; ++i) {
            const unsigned sq = seq0 + i, par = sq & 1u;
            if (i < most) {
                const ulonglong2* wx = I.lowx + (size_t)par * 3 * n;
                double v[2];
                bool want[2];
                const ulonglong2* p[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int t = tid - 32 + 64 * h, r = t / 3;
                    const int k = r < kHalo ? s - kHalo + r : e + 1 + (r - kHalo);
                    want[h] = t < 6 * kHalo && k >= 0 && k < n && K > 1;
                    p[h] = wx + (want[h] ? 3 * (size_t)k + (t - 3 * r) : 0);
                    v[h] = 0.0;
                }
                unsigned long long it = 0;
                for (;;) {
                    bool there = true;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (want[h]) there &= ld_tagged(p[h], sq, v[h]);
                    if (there) break;
                    if (++it > limit) {
                        *(volatile int*)&C.lo_fail = 1;
                        break;
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int t = tid - 32 + 64 * h, r = t / 3;
                    if (t < 6 * kHalo) C.halo[par][r][t - 3 * r] = v[h];
                }
                __syncwarp();
            }
            if (i > 0) {
                bar_told();
                if (*(volatile int*)&C.lo_state[0] != kLoGoOn) break;
            }
            bar_rows();
        }
    } else if (warp == 3) {
        // the residuals of all chunks
        for (int i = 0;; ++i) {
            const unsigned sq = seq0 + i;
            const ulonglong2* lr = I.lores + (size_t)(sq & 3u) * K * 2;
            double a = 0.0;
            bool fl = false;
            for (int j = lane; j < K; j += 32) {
                double y;
                unsigned long long it = 0;
                while (!ld_tagged(lr + j, sq, y)) {
                    if (++it > limit) {
                        *(volatile int*)&C.lo_fail = 1;
                        break;
                    }
                }
                fl |= y < 0.0;
                a = __double_as_longlong(fabs(y)) > __double_as_longlong(a) ? fabs(y) : a;
            }
            __syncwarp();
            fl = __any_sync(0xffffffffu, fl);
            a = rows::warp_max_bits(a);
            if (lane == 0) C.lres[sq & 1u] = fl ? -1.0 : a;
            __syncwarp();
            bar_res();
            bar_told();
            if (*(volatile int*)&C.lo_state[0] != kLoGoOn) break;
        }
    }
    __syncthreads();
    seq = C.lo_seq[0];
    out.max_y = my;
    if (C.lo_state[0] == kLoFailed) return false;
    out.iters = C.lo_state[1];
    out.std_res = C.lo_std;
    out.df = -1.0;  // in the residual records of exchange out.seq
    out.seq = C.lo_seq[1];
    if (C.lo_state[0] == kLoGeneral) {
        const int m0 = C.lo_state[1];
        __syncthreads();
        return lo_general(C, scratch, c, z, m0, seq, limit, out);
    }
    return true;
}

// Phase trace: end of one phase, start of another (slots of trace_h, -1: none).  Not
// inlined: the marks' code in the kernel cost 2% of a step without a trace.
static __device__ __noinline__ void mark(const HoloDev& P, int z, int end, int start) {
    if (end >= 0) trace_h(P, z, end, false);
    if (start >= 0) trace_h(P, z, start, true);
}
static __device__ __noinline__ void mark_lo(const HoloDev& P, int z, int lo_iters) {
    mark(P, z, 11, -1);
    mark(P, z, 3, -1);
    if (blockIdx.x == 0 && threadIdx.x == 0 && 4 * z + 3 < P.head.trace_iters)
        P.head.trace[(size_t)16 * z + 6] = (unsigned long long)lo_iters;
}

__global__ void __launch_bounds__(512, 1) holo_rows_kernel(HoloDev* __restrict__ Pp, int swap_io) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HoloDev& P = *Pp;
    HoloSmem& C = *reinterpret_cast<HoloSmem*>(smem_raw);
    const HoloInst& I = C.I;
    const unsigned long long limit = P.head.spin_limit;
    const bool traced = P.head.trace != nullptr;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const int b = find_inst(P.blk_off, P.n_inst, (long long)blockIdx.x);
    const int blk = (int)((long long)blockIdx.x - __ldg(&P.blk_off[b]));
    {
        const int* s = reinterpret_cast<const int*>(&P.inst[b]);
        int* d = reinterpret_cast<int*>(&C.I);
        for (int q = tid; q < (int)(sizeof(HoloInst) / sizeof(int)); q += blockDim.x) d[q] = __ldg(s + q);
        if (tid == 0) {
            C.bad[0] = C.bad[1] = C.lo_fail = 0;
            C.set = rows::launch_parity(&P.arrivals, gridDim.x);
        }
    }
    __syncthreads();
    double* const misc = I.misc + 4 * C.set;
    if (blk == 0 && tid < 4) I.misc[4 * (C.set ^ 1) + tid] = 0.0;
    const int nt_max = I.nt_neg > I.nvt - I.nt_neg ? I.nt_neg : I.nvt - I.nt_neg;
    const int nslot = nt_max < kSignSlots ? nt_max : kSignSlots;
    TileBuf* bufs = reinterpret_cast<TileBuf*>(smem_raw + sizeof(HoloSmem));
    double(*part)[4][32] = reinterpret_cast<double(*)[4][32]>(bufs + nw);  // [sign][slot]
    unsigned char* scratch = reinterpret_cast<unsigned char*>(bufs);
    const double* fn = swap_io ? I.f_out : I.f_in;
    double* fo = swap_io ? const_cast<double*>(I.f_in) : I.f_out;
    const int k0 = blk * I.rblk;
    const int nr = I.n_inner - k0 < I.rblk ? I.n_inner - k0 : I.rblk;
    rows::TaggedMaps maps{{I.maps, I.maps}, 0u, nullptr, 0};
    ulonglong2* const horec = I.horec;

    // ---- prologue
    if (blk == 0 && tid == 0) {
        I.stats->status = KEQ_ERR_TIMEOUT;  // pending until the statistics
        if (P.head.fresh) {
            I.stats->total_iters = 0;
            I.stats->total_steps = 0;
        }
    }
    // tags of the launch before
    for (int vt = warp; vt < I.nvt; vt += nw) {
        ulonglong2* p = maps.slot(I, 0, blk, vt);
        st_tagged(p, 0.0, 0u);
        st_tagged(p + 32, 0.0, 0u);
    }
    if (tid < 8) st_tagged(horec + ((size_t)(tid >> 2) * I.nblk + blk) * 4 + (tid & 3), 0.0, 0u);
    for (int t = tid; t < nr * 12; t += blockDim.x) st_tagged(I.rowd + 12 * (size_t)(k0 + 1) + t, 0.0, 0u);
    for (int t = tid; t < nr * 4; t += blockDim.x) st_tagged(I.wlo + 4 * (size_t)(k0 + 1) + t, 0.0, 0u);
    for (int t = tid; t < nr * 6; t += blockDim.x)
        st_tagged(I.lowx + (size_t)(t / (nr * 3)) * 3 * I.n_inner + 3 * (size_t)k0 + t % (nr * 3), 0.0, 0u);
    if (blk < I.lo_n && tid == 9) st_tagged(I.loy + blk, 0.0, 0u);
    if (blk < I.lo_n && tid < 9)
        st_tagged(tid < 8 ? I.lores + (size_t)(tid >> 1) * I.lo_n * 2 + (size_t)(tid & 1) * I.lo_n + blk : I.locm + blk,
                  0.0, 0u);
    if (blk < I.lo_n)
        for (int t = tid; t < 2 * kLoRec; t += blockDim.x)
            st_tagged(I.lorec + ((size_t)(t / kLoRec) * I.lo_n + blk) * kLoRec + t % kLoRec, 0.0, 0u);
    // raw half-range sums of f^n
    for (int vt = warp; vt < I.nvt; vt += nw) {
        TileBuf& w = bufs[warp];
        const Tile g = rows::make_tile(I, blk, vt);
        rows::copy_tile(I, w, g, fn);
        cp_async_wait_all();
        const double vj = w.vw[lane].x;
        w.vw[lane].y = vj * vj;
        __syncwarp();
        bool first;
        const int sl = slot_of(I, nslot, vt, first);
        rows::row_sums<4>(w, g, I.rblk, first, part[sl]);
        __syncwarp();
    }
    if (blk == 0 && warp == nw - 1) boundary_row_h(I, fn, fo, 0, misc);
    if (blk == I.nblk - 1 && warp == nw - 2) boundary_row_h(I, fn, fo, 1, misc);
    __syncthreads();
    if (warp == 0 && lane < nr) {
        const int i = k0 + lane + 1;
        double R8[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            R8[q] = half_sum(I, part, nslot, q);
            C.R[lane][q] = R8[q];
            I.Rn[8 * (size_t)i + q] = R8[q];
        }
        const Mom m = mom_nr(R8, I.dv);
        double c4[4];
        mc_nr(m.n, m.u, m.T, I.tau_tilde, c4);
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
            for (int q = 0; q < 4; ++q) C.coef[d][d == 0 ? lane : nr - 1 - lane][q] = c4[q];
        // W_HO = (n, n u, n (u^2 + T) / 2) (:268-271)
        I.Who[3 * (size_t)i + 0] = m.n;
        I.Who[3 * (size_t)i + 1] = m.n * m.u;
        I.Who[3 * (size_t)i + 2] = 0.5 * m.n * (m.u * m.u + m.T);
    }
    __syncthreads();
    // explicit term, Maxwellian sums of f^n
    double emax = 0.0;
    for (int vt = warp; vt < I.nvt; vt += nw) {
        TileBuf& w = bufs[warp];
        const Tile g = rows::make_tile(I, blk, vt);
        rows::copy_tile(I, w, g, fn);
        const double em = explicit_tile_h(C, w, g, fn);
        emax = em > emax ? em : emax;
        bool first;
        const int sl = slot_of(I, nslot, vt, first);
        rows::row_sums<3>(w, g, I.rblk, first, part[sl]);
        __syncwarp();
    }
    emax = rows::warp_max_bits(emax);
    if (lane == 0) atomic_max_nonneg(&misc[2], emax);
    __syncthreads();
    if (warp == 0 && lane < nr) {
        // I_old = (1-theta) (sum M_old w - sum f^n w) dv / tau_old
        const int i = k0 + lane + 1;
        const Mom m = mom_nr(C.R[lane], I.dv);
        const double inv_tau = C.coef[0][lane][3];
        double sM[3];
#pragma unroll
        for (int q = 0; q < 3; ++q)
            sM[q] = half_sum(I, part, nslot, q) + half_sum(I, part, nslot, 4 + q);
        const double smw[3] = {sM[0] * I.dv, sM[1] * I.dv, 0.5 * (sM[2] * I.dv)};
        const double sfw[3] = {m.n, m.s1, 0.5 * m.s2};
#pragma unroll
        for (int q = 0; q < 3; ++q)
            I.Iold[3 * (size_t)i + q] = (1.0 - kTheta) * ((smw[q] - sfw[q]) * inv_tau);
    }
    if (!rows::launch_barrier(&P.arrivals, gridDim.x, limit)) {
        if (tid == 0) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
        return;
    }
    const double bmax = __ldcg(&misc[0]);
    const double gconst = fmax(__ldcg(&misc[2]), bmax);
    if (tid < 16) C.Rb[tid >> 3][tid & 7] = __ldcg(&I.Rn[8 * (size_t)(tid < 8 ? 0 : I.nx - 1) + (tid & 7)]);
    if (warp < I.nvt) rows::copy_tile(I, bufs[warp], rows::make_tile(I, blk, warp), I.E);

    double ho_std = 0.0, ho_df = 0.0, ho_ref = 0.0;
    bool bad_last = false, failed = false;
    LoResult lo{};
    unsigned seq = 0;
    int z = 0;
    for (;; ++z) {
        const unsigned tag = (unsigned)z + 1u;
        bool ok = true;
        __syncthreads();  // C.R is complete
        if (traced) mark(P, z, -1, 0);
        // A: velocity sums of M(f_z) per row, a row per warp
        if (I.con_terms)
            for (int r = warp; r < nr; r += nw) {
                const Mom m = mom_nr(C.R[r], I.dv);
                double c4[4], s3[3];
                mc_nr(m.n, m.u, m.T, I.tau_tilde, c4);
                maxwell_sums4(I.v, I.nv, c4, s3);
                if (lane < 3) {
                    const double t = lane == 0 ? s3[0] : (lane == 1 ? s3[1] : s3[2]);
                    st_tagged(I.rowd + 12 * (size_t)(k0 + r + 1) + 8 + lane, t, tag);
                }
            }
        else
            for (int t = tid; t < nr * 3; t += blockDim.x)
                st_tagged(I.rowd + 12 * (size_t)(k0 + t / 3 + 1) + 8 + t % 3, 0.0, tag);
        for (int t = tid; t < nr * 8; t += blockDim.x)
            st_tagged(I.rowd + 12 * (size_t)(k0 + (t >> 3) + 1) + (t & 7), C.R[t >> 3][t & 7], tag);
        if (traced) mark(P, z, 1, 2);
        if (blk < I.lo_n) {
            cp_async_wait_all();
            __syncthreads();
            if (traced) mark(P, z, -1, 8);
            ok = lo_solve(C, scratch, blk, z, seq, limit, lo);
            if (traced) mark(P, z, 9, -1);
            if (tid == 0) st_tagged(I.loy + blk, lo.max_y, tag);
            // (the general interface solve may have used the tile buffers)
            if (warp < I.nvt) rows::copy_tile(I, bufs[warp], rows::make_tile(I, blk, warp), I.E);
        }
        // LO solution of the block's rows and the largest coefficient of all chunks
        if (traced) mark(P, z, -1, 10);
        {
            double cm = 0.0;
            for (int t = tid; t < nr * 3 + I.lo_n; t += blockDim.x) {
                const bool row = t < nr * 3;
                const ulonglong2* p = row ? I.wlo + 4 * (size_t)(k0 + 1 + t / 3) + t % 3 : I.locm + (t - nr * 3);
                double v = 0.0;
                unsigned long long it = 0;
                while (ok && !ld_tagged(p, tag, v)) {
                    if (++it > limit) ok = false;
                    if (it < 1000000ull) __nanosleep(100);  // the LO iteration takes tens of us
                }
                if (row) C.Wl[t / 3][t % 3] = v;
                else cm = __double_as_longlong(v) > __double_as_longlong(cm) ? v : cm;
            }
            __syncwarp();
            cm = rows::warp_max_bits(cm);
            if (lane == 0) C.cmax[warp] = cm;
        }
        if (!__syncthreads_and(ok)) {
            failed = true;
            break;
        }
        if (traced) mark_lo(P, z, lo.iters);
        if (warp == 0 && lane < nr) {
            const int i = k0 + lane + 1;
            double u, T, c4[4];
            lo_state(C.Wl[lane], u, T);
            mc_nr(C.Wl[lane][0], u, T, I.tau_tilde, c4);
            c4[3] = (kTheta * I.dt) * c4[3];
            rows::put_coef(C, lane, nr, c4);
            I.Wlo[i] = C.Wl[lane][0];
            I.Wlo[I.nx + i] = u;
            I.Wlo[2 * (size_t)I.nx + i] = T;
        }
        const double G = fmax(gconst, 1.0000001 * rows::warp_max_bits(lane < nw ? C.cmax[lane] : 0.0));
        __syncthreads();
        // C: distribution sweep
        if (traced) mark(P, z, -1, 4);
        maps.tag = tag;
        HoResidual pr(I.ho_tol, I.ho_abs_tol);
        bool bad = false;
        for (int vt = warp; vt < I.nvt; vt += nw) {
            const Tile g = rows::make_tile(I, blk, vt);
            bool first;
            const int sl = slot_of(I, nslot, vt, first);
            ok &= rows::sweep_tile<true, 4>(C, bufs[warp], part[sl], first, g, blk, vt, z, I.dtdx2, G, maps,
                                            limit, fn, fo, pr, bad);
            // the next tile, behind the last one the first of the next iteration
            rows::copy_tile(I, bufs[warp], rows::make_tile(I, blk, vt + nw < I.nvt ? vt + nw : warp), I.E);
        }
        {
            double r1 = pr.q1.special != pr.q1.special || pr.q1.special > 0.0
                            ? pr.q1.value() : div_nr(pr.q1.num, pr.q1.den);
            r1 = rows::warp_max_bits(r1);
            const double r2 = rows::warp_max_bits(pr.mdf), r3 = rows::warp_max_bits(pr.mref);
            if (lane == 0) {
                C.red[warp][0] = r1;
                C.red[warp][1] = r2;
                C.red[warp][2] = r3;
            }
        }
        // (as numbers a give-up is above the rest, so that the largest of all blocks tells)
        const int flags = (__any_sync(0xffffffffu, bad) ? kBadValue : 0) | (__any_sync(0xffffffffu, !ok) ? kBadWait : 0);
        if (flags != 0 && lane == 0) atomicOr(&C.bad[z & 1], flags);
        if (traced) mark(P, z, 5, 12);
        __syncthreads();
        ulonglong2* recs = horec + (size_t)(z & 1) * I.nblk * 4;
        if (warp == 0) {
            double v[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) v[q] = rows::warp_max_bits(lane < nw ? C.red[lane][q] : 0.0);
            if (lane < 4)
                st_tagged(recs + 4 * (size_t)blk + lane,
                          lane == 0 ? v[0] : lane == 1 ? v[1] : lane == 2 ? v[2] : (double)C.bad[z & 1], tag);
            __syncwarp();
            if (lane == 0) C.bad[(z & 1) ^ 1] = 0;
        }
        // raw sums of f_{z+1}: a quantity per warp
        for (int q = warp; q < 8; q += nw) {
            const double v = half_sum(I, part, nslot, q);
            if (lane < nr) C.R[lane][q] = v;
        }
        {
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            int t0 = tid - 32;
            if (t0 < 0) t0 += blockDim.x;
            for (int t = t0; t < I.nblk; t += blockDim.x) {
                const ulonglong2* p = recs + 4 * (size_t)t;
                double a[4];
                unsigned long long it = 0;
                for (;;) {
                    bool there = true;
#pragma unroll
                    for (int q = 0; q < 4; ++q) there &= ld_tagged(p + q, tag, a[q]);
                    if (there) break;
                    if (++it > limit) {
                        ok = false;
                        break;
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    v[q] = __double_as_longlong(a[q]) > __double_as_longlong(v[q]) ? a[q] : v[q];
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                v[q] = rows::warp_max_bits(v[q]);
                if (lane == 0) C.all[z & 1][warp][q] = v[q];
            }
        }
        if (!__syncthreads_and(ok)) {
            failed = true;
            break;
        }
        ho_std = rows::warp_max_bits(lane < nw ? C.all[z & 1][lane][0] : 0.0);
        ho_df = rows::warp_max_bits(lane < nw ? C.all[z & 1][lane][1] : 0.0);
        ho_ref = rows::warp_max_bits(lane < nw ? C.all[z & 1][lane][2] : 0.0);
        if (traced) mark(P, z, 13, -1);
        const double worst = rows::warp_max_bits(lane < nw ? C.all[z & 1][lane][3] : 0.0);
        if (worst >= kBadWait) {
            failed = true;
            break;
        }
        bad_last = worst != 0.0;
        if (I.fixed_ho > 0 ? z + 1 >= I.fixed_ho : ho_std <= 1.0) break;
        if (z + 1 >= I.ho_iter) break;
    }
    cp_async_wait_all();
    if (failed) {
        if (tid == 0) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
        return;
    }
    if (blockIdx.x == 0 && tid == 0) P.head.fresh = 0;
    bool done = true;  // (a wait below that gives up leaves the pending status)
    if (blk == 0 && warp == 0) {
        // the largest |Y| of the step's last HO iteration, and the LO difference
        // of the windows, from the chunks' records
        double df = 0.0, my = 0.0;
        for (int t = lane; t < I.lo_n; t += 32) {
            double v;
            unsigned long long it = 0;
            if (lo.df < 0.0) {
                const ulonglong2* p = lo.df == -1.0
                                          ? I.lores + (size_t)(lo.seq & 3u) * I.lo_n * 2 + I.lo_n + t
                                          : I.lorec + ((size_t)(lo.seq & 1u) * I.lo_n + t) * kLoRec + kRecDf;
                while (!ld_tagged(p, lo.seq, v))
                    if (++it > limit) {
                        done = false;
                        break;
                    }
                df = __double_as_longlong(v) > __double_as_longlong(df) ? v : df;
            }
            while (!ld_tagged(I.loy + t, (unsigned)z + 1u, v))
                if (++it > limit) {
                    done = false;
                    break;
                }
            my = __double_as_longlong(v) > __double_as_longlong(my) ? v : my;
        }
        __syncwarp();
        df = rows::warp_max_bits(df);
        lo.max_y = rows::warp_max_bits(my);
        if (lo.df < 0.0) lo.df = df;
        done = __all_sync(0xffffffffu, done);
        if (!done && lane == 0) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
    }
    if (blk == 0 && tid == 0 && done) {
        keq_step_stats* st = I.stats;
        st->status = bad_last ? KEQ_ERR_NONFINITE : KEQ_OK;
        st->iters = z + 1;
        st->aa_applied = 0;
        st->lo_iters = lo.iters;
        st->residual = ho_df / nan_max(ho_ref, bmax);
        st->std_residual = ho_std;
        st->lo_residual = lo.df;
        st->std_lo_residual = lo.std_res;
        st->max_YI = lo.max_y;
        st->total_iters += z + 1;
        st->total_steps += 1;
    }
}

}  // namespace holo

const void* holo_rows_entry() { return (const void*)holo::holo_rows_kernel; }
// nslot: partial-sum slots per sign of v; lo_n: LO chunks (the general interface
// solve works in the tile buffers and the slots).
size_t holo_rows_smem(int warps, int nslot, int lo_n) {
    const size_t work = (size_t)warps * sizeof(rows::TileBuf) + (size_t)2 * nslot * 4 * 32 * sizeof(double);
    const int g = (lo_n + 31) / 32;
    const size_t lo = sizeof(holo::GroupRec) * g + 13 * sizeof(double) * (size_t)lo_n + 3 * sizeof(double) * g;
    return sizeof(holo::HoloSmem) + (work > lo ? work : lo);
}
size_t holo_rows_lorec_units(int lo_n) { return 2 * (size_t)lo_n * holo::kLoRec; }

}  // namespace keq
