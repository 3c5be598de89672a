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
// What bounds it: instruction issue inside the sweep (about 150 issue cycles
// per row of 32 cells and scheduler, 60 of them FP64) and, for small grids,
// the dependent latencies of one iteration (publish, fold, row sums, update,
// barrier).  Measured against the look-back kernel on one B200, us per step:
// 4096x512 812 -> 354, 8192x1024 1772 -> 862, 256x128 319 -> 142.
//
// Bounds.  x_i is a convex combination of f^n_i, M_i and x_{i-1} (weights
// 1/d, (dt/tau)/d, cpl/d with d = 1 + dt/tau + cpl), so no |x| exceeds
// G = max(max |f^n|, max M), and a_i = cpl/d <= cpl/(1 + cpl) < 1.  Plan
// creation admits an instance to this kernel when a product of a_max over at
// most kmax blocks is below 2^-200; beyond that the look-back kernel runs.
#include <cuda_runtime.h>
#include <stddef.h>

#include "keq_common.cuh"
#include "keq_implicit.cuh"
#include "keq_internal.h"

namespace keq {
namespace rows {

constexpr int kRows = KEQ_ROWS_MAX;
constexpr int kFold = 4;       // maps that a fold loads at a time
constexpr int kListMax = 512;  // instances of a plan that the active list holds
constexpr int kSlots = 16;  // partial-sum slots: v-tile vt adds into slot vt & 15
constexpr unsigned long long kEmptyBits = ~0ull;  // map not published yet (a NaN no arithmetic makes)

struct TileBuf {
    double a[kRows][33];  // f^n, then Y of the zero-inflow recurrence, then x, in scan order
    double2 vw[32];       // (v, v^2) of the tile's lanes
};

struct alignas(16) CtaSmem {
    ImpInst I;
    // u, -1/(2T), dt/tau n/sqrt(2 pi T), dt/tau per row, in both scan orders
    alignas(16) double coef[2][kRows][4];
    double red[kSlots][2];
    double gbound, nm;
    double gs[kMaxPairs];  // Gram matrix
    unsigned next[2];  // claimed list position, by parity of the claim
    int n_act, act_items;  // active instances of the iteration and their items
    int bad;
    int ok;  // outcome of the grid barrier
};

// Anderson history of the rows of one instance's block (solo plans): residual
// and moment columns.
struct Ring {
    double R[kMaxAACols][3][32], G[kMaxAACols][3][32];
};

// read as double2
static_assert(offsetof(CtaSmem, coef) % 16 == 0 && sizeof(CtaSmem) % 16 == 0, "alignment");
static_assert(offsetof(TileBuf, vw) % 16 == 0 && sizeof(TileBuf) % 16 == 0, "alignment");

__device__ __forceinline__ double2 ld_map(const double2* p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_map(double2* p, double x, double y) {
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(x), "d"(y) : "memory");
}
__device__ __forceinline__ bool is_empty(double v) {
    return (unsigned long long)__double_as_longlong(v) == kEmptyBits;
}
// A value that happens to carry the empty pattern is published as another NaN.
__device__ __forceinline__ double not_empty(double v) {
    return is_empty(v) ? __longlong_as_double(0x7ff8000000000000ll) : v;
}

// e^x for x <= 0 as exp_nonpos (keq_common.cuh), with results below 2^-1021
// flushed to zero and the scale 2^k added to the exponent field, which saves
// two FP64 operations and the compare of the clamp.
__device__ __forceinline__ double exp_neg(double x) {
    constexpr double LOG2E = 1.4426950408889634;
    constexpr double LN2_HI = 0.6931471806019545;
    constexpr double LN2_LO = -4.2009150726810846e-11;
    constexpr double ROUND = 6755399441055744.0;  // 1.5 * 2^52
    // clamp at about -746 by the high word (as unsigned, more negative is larger)
    unsigned hx = (unsigned)__double2hiint(x);
    hx = hx < 0xC0875000u ? hx : 0xC0875000u;
    const double xc = __hiloint2double((int)hx, __double2loint(x));
    const double kr = fma(xc, LOG2E, ROUND);
    const int ki = __double2loint(kr);
    const double k = kr - ROUND;
    double r = fma(-k, LN2_HI, xc);
    r = fma(-k, LN2_LO, r);
    double p = 1.6059043836821613e-10;
    p = fma(p, r, 2.08767569878681e-09);
    p = fma(p, r, 2.505210838544172e-08);
    p = fma(p, r, 2.755731922398589e-07);
    p = fma(p, r, 2.7557319223985893e-06);
    p = fma(p, r, 2.48015873015873e-05);
    p = fma(p, r, 0.0001984126984126984);
    p = fma(p, r, 0.001388888888888889);
    p = fma(p, r, 0.008333333333333333);
    p = fma(p, r, 0.041666666666666664);
    p = fma(p, r, 0.16666666666666666);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = fma(p, r, 1.0);
    const bool z = ki < -1021;
    const int hi = z ? 0 : __double2hiint(p) + (ki << 20);
    const int lo = z ? 0 : __double2loint(p);
    return __hiloint2double(hi, lo);
}

// One tile: 32 velocities (lane) x the block's rows.  Scan position r runs
// along the characteristics: row r of the block for v > 0, row nr-1-r else.
// Lanes past the last (before the first) velocity of a sign repeat the nearest
// one, so that they need no masks; their rows are not stored nor summed.
struct Tile {
    bool pos, lane_ok;
    int j;         // velocity of the lane (clamped)
    int lo, hi;    // lanes [lo, hi) hold the tile's velocities
    int k0, nr;    // first interior row and rows of the block
    int st;        // elements from one scan position to the next
    size_t first;  // element of scan position 0
};

__device__ __forceinline__ Tile make_tile(const ImpInst& I, int blk, int vt) {
    const int lane = threadIdx.x & 31;
    Tile t;
    t.pos = vt >= I.nt_neg;
    if (t.pos) {
        const int j0 = I.kp + 32 * (vt - I.nt_neg);
        t.lo = 0;
        t.hi = I.nv - j0 < 32 ? I.nv - j0 : 32;
        t.j = j0 + (lane < t.hi ? lane : t.hi - 1);
    } else {
        const int j0 = I.kp - 32 * (vt + 1);
        t.lo = j0 < 0 ? -j0 : 0;
        t.hi = 32;
        t.j = j0 + (lane < t.lo ? t.lo : lane);
    }
    t.lane_ok = lane >= t.lo && lane < t.hi;
    t.k0 = blk * I.rblk;
    t.nr = I.n_inner - t.k0 < I.rblk ? I.n_inner - t.k0 : I.rblk;
    t.st = t.pos ? I.nv : -I.nv;
    t.first = (size_t)(t.pos ? 1 + t.k0 : t.k0 + t.nr) * I.nv + t.j;
    return t;
}

__device__ __forceinline__ double2* map_slot(const ImpInst& I, int par, int blk, int vt) {
    return I.xch + (((size_t)par * I.nblk + blk) * I.nvt + vt) * 32 + (threadIdx.x & 31);
}

// Start the copy of the tile's f^n (scan order) and velocities into shared
// memory; lane copies its own column.
__device__ __forceinline__ void copy_tile(const ImpInst& I, TileBuf& w, const Tile& g,
                                          const double* __restrict__ fn) {
    const int lane = threadIdx.x & 31;
    const double* p = fn + g.first;
    double* d = &w.a[0][lane];
    cp_async8(&w.vw[lane].x, &I.v[g.j]);
#pragma unroll 4
    for (int r = 0; r < g.nr; ++r) {
        cp_async8(d, p);
        d += 33;
        p += g.st;
    }
    cp_async_commit();
}

__device__ __forceinline__ void ld4(double (&d)[4], const double* p, long long st) {
#pragma unroll
    for (int t = 0; t < 4; ++t) d[t] = __ldcg(p + t * st);
}

// Largest of the lanes' values, each non-negative or +NaN (which wins): their
// bit patterns order like unsigned integers.
__device__ __forceinline__ double warp_max_bits(double v) {
    const unsigned hi = (unsigned)__double2hiint(v);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)__double2loint(v) : 0u);
    return __hiloint2double((int)mh, (int)ml);
}

// Inflow of the tile's lanes: X = Y_1 + P_1 (Y_2 + P_2 (...)) over the blocks
// upstream (1 = nearest), down to the boundary value.  With p the product of
// the P so far and G a bound of every |x|, the terms left out are below p G;
// the fold ends when, for every lane, that is below 2^-58 of max(|X|, abs_tol)
// or 2^-200 of G.  The number of blocks folded depends on the data alone, so
// the result does not depend on timing.  False if a wait gave up.
__device__ __forceinline__ bool fold_carry(const ImpInst& I, const Tile& g, const double* fn,
                                           int par, int blk, int vt, double G,
                                           unsigned long long limit, double& X) {
    const double eps = 3.469446951953614e-18;                 // 2^-58
    const double floor_g = G * 6.223015277861142e-61;         // 2^-200
    const int avail = g.pos ? blk : I.nblk - 1 - blk;         // blocks upstream
    const int last = avail < I.kmax ? avail : I.kmax;
    const double2* p0 = map_slot(I, par, blk, vt);
    const long long step = (long long)(g.pos ? -1 : 1) * I.nvt * 32;
    double acc = 0.0, pr = 1.0;
    const double amin = I.abs_tol;
    for (int k = 1; k <= last; k += kFold) {
        // kFold blocks in flight together (past the last one: the last again)
        double2 v[kFold];
        unsigned long long it = 0;
        for (;;) {
            bool miss = false;
#pragma unroll
            for (int t = 0; t < kFold; ++t) {
                v[t] = ld_map(p0 + (k + t < last ? k + t : last) * step);
                miss |= is_empty(v[t].x) || is_empty(v[t].y);
            }
            if (!__any_sync(0xffffffffu, miss)) break;
            if (++it > limit) {
                X = acc;
                return false;
            }
        }
#pragma unroll
        for (int t = 0; t < kFold; ++t) {
            if (k + t <= last) {
                acc = fma(pr, v[t].y, acc);
                pr *= v[t].x;
                const double aa = fabs(acc) > amin ? fabs(acc) : amin;
                const double th = eps * aa > floor_g ? eps * aa : floor_g;
                if (!__any_sync(0xffffffffu, !(pr * G <= th))) {
                    X = acc;
                    return true;
                }
            }
        }
    }
    if (last == avail)  // the boundary row is the inflow of the first block
        acc = fma(pr, __ldcg(&fn[(size_t)(g.pos ? 0 : I.nx - 1) * I.nv + g.j]), acc);
    X = acc;
    return true;
}

// Sums over the tile's velocities of x (1, v, v^2) per row, added to (first
// tile of the slot: stored into) part[slot].  Lane = row; with 8 or 16 rows
// the columns are split over 4 or 2 lanes per row and combined by shuffles.
// Returns whether the lane's sum of x is finite.
__device__ __forceinline__ bool row_sums(const TileBuf& w, const Tile& g, int rblk, int vt,
                                         double (*part)[3][32]) {
    const int lane = threadIdx.x & 31;
    const int w2 = rblk <= 8 ? 8 : (rblk <= 16 ? 16 : 32);  // lanes per column group
    const int r = lane & (w2 - 1), grp = lane / w2;
    const int per = w2;  // 32 / (32 / w2) columns per group
    int j = grp * per, je = j + per;
    j = j > g.lo ? j : g.lo;
    je = je < g.hi ? je : g.hi;
    // four running sums per quantity (columns j, j+1, j+2, j+3 of every four):
    // a single one would wait for 32 dependent additions
    double q0[4], q1[4], q2[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) q0[c] = q1[c] = q2[c] = 0.0;
    if (r < g.nr) {
        const double* a = w.a[g.pos ? r : g.nr - 1 - r];
#pragma unroll 2
        for (; j + 4 <= je; j += 4) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double x = a[j + c];
                const double2 vv = w.vw[j + c];
                q0[c] += x;
                q1[c] = fma(x, vv.x, q1[c]);
                q2[c] = fma(x, vv.y, q2[c]);
            }
        }
        for (; j < je; ++j) {
            const double x = a[j];
            const double2 vv = w.vw[j];
            q0[0] += x;
            q1[0] = fma(x, vv.x, q1[0]);
            q2[0] = fma(x, vv.y, q2[0]);
        }
    }
    double s0 = (q0[0] + q0[1]) + (q0[2] + q0[3]);
    double s1 = (q1[0] + q1[1]) + (q1[2] + q1[3]);
    double s2 = (q2[0] + q2[1]) + (q2[2] + q2[3]);
    for (int o = w2; o < 32; o <<= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane < w2) {
        double(*p)[32] = part[vt & (kSlots - 1)];
        if (vt >= kSlots) {
            s0 += p[0][r];
            s1 += p[1][r];
            s2 += p[2][r];
        }
        p[0][r] = s0;
        p[1][r] = s1;
        p[2][r] = s2;
    }
    return isfinite(s0);
}

// Row sum of quantity q over all tiles from the slots (lane = row), in four
// running sums.
__device__ __forceinline__ double slot_sum(const double (*part)[3][32], int nvt, int q) {
    const int lane = threadIdx.x & 31;
    const int ns = nvt < kSlots ? nvt : kSlots;
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    for (int t = 0; t < ns; t += 4) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double v = part[t + c < ns ? t + c : t][q][lane];
            a[c] += t + c < ns ? v : 0.0;
        }
    }
    return (a[0] + a[1]) + (a[2] + a[3]);
}

__device__ __forceinline__ bool inst_active_rows(const ImpInst& I, int m) {
    if (m >= I.picard_iter) return false;
    if (I.fixed_iters > 0) return m < I.fixed_iters && inst_enabled(I);
    if (m == 0) return inst_enabled(I);
    // a slot is zero until its iteration has run, so an instance that stopped
    // (or is switched off) stays inactive
    return !(ld_cg(&I.res[2 * (m - 1)]) <= 1.0);
}

// ---- one Picard sweep of one tile -------------------------------------------
// Residual |x - o| / (abs_tol + tol ref) and |x - o| / max(ref, abs_tol),
// ref = max(|x|, |o|), into the running maxima.  With abs_tol > 0 and finite
// x the denominators are positive; `strict` (abs_tol or tol not positive)
// takes the general update.  Non-finite x are found from the row sums.
__device__ __forceinline__ void residual(double x, double o, double tol, double abs_tol, bool strict,
                                         FracMax& q1, FracMax& q2) {
    const double df = fabs(x - o);
    const double ref = fabs(x) > fabs(o) ? fabs(x) : fabs(o);
    const double b1 = fma(tol, ref, abs_tol);
    const double b2 = ref > abs_tol ? ref : abs_tol;
    if (strict) {
        q1.add(df, b1);
        q2.add(df, b2);
    } else {
        const bool t1 = df * q1.den > q1.num * b1, t2 = df * q2.den > q2.num * b2;
        q1.num = t1 ? df : q1.num;
        q1.den = t1 ? b1 : q1.den;
        q2.num = t2 ? df : q2.num;
        q2.den = t2 ? b2 : q2.den;
    }
}

// Values of both running maxima, the two quotients interleaved.
__device__ __forceinline__ void frac_values(const FracMax& q1, const FracMax& q2, double& v1, double& v2) {
    if (q1.den >= 1e-270 && q1.den <= 1e270 && q2.den >= 1e-270 && q2.den <= 1e270) {
        const double r1 = recip3(q1.den), r2 = recip3(q2.den);
        const double a = q1.num * r1, b = q2.num * r2;
        v1 = fma(fma(-a, q1.den, q1.num), r1, a);
        v2 = fma(fma(-b, q2.den, q2.num), r2, b);
    } else {
        v1 = q1.num / q1.den;
        v2 = q2.num / q2.den;
    }
    // a quotient met on the general path (NaN wins)
    v1 = v1 > q1.special ? v1 : q1.special;
    v2 = v2 > q2.special ? v2 : q2.special;
}

// The tile's f^n is in (or on its way to) w.a.
template <bool kResidual>
__device__ __forceinline__ bool sweep_tile(const CtaSmem& C, TileBuf& w, double (*part)[3][32],
                                           const Tile& g, int blk, int vt, int m, double G,
                                           unsigned long long limit, const double* __restrict__ fn,
                                           double* __restrict__ fo, FracMax& q1, FracMax& q2,
                                           bool& bad) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int nr = g.nr, nr4 = nr & ~3;
    const double(*co)[4] = C.coef[g.pos ? 0 : 1];
    double* col = &w.a[0][lane];
    cp_async_wait_all();
    const double vj = w.vw[lane].x;
    w.vw[lane].y = vj * vj;
    const double cpl = I.dtdx * fabs(vj);
    const double one_plus = 1.0 + cpl;
    // The recurrence starts from the previous iterate's inflow X0 instead of
    // zero, so that what is left to correct, the product of the a times
    // (X - X0), dies out sooner (the iterates converge).
    const long long st = g.st;
    const double* po = (m > 0 ? fo : fn) + g.first;
    const double X0 = __ldcg(po - st);
    double P = 1.0, Y = X0;
    int neg = __double2hiint(X0);
    auto assemble = [&](int r, double& av, double& cv) {
        const double2 ca = *reinterpret_cast<const double2*>(co[r]);
        const double2 cb = *reinterpret_cast<const double2*>(co[r] + 2);
        const double diff = vj - ca.x;
        const double e = exp_neg(diff * diff * ca.y);
        const double rr = recip3(one_plus + cb.y);
        cv = fma(cb.x, e, col[33 * r]) * rr;
        av = cpl * rr;
    };
    auto advance = [&](int r, double av, double cv) {
        Y = fma(av, Y, cv);
        P = P * av;
        neg |= __double2hiint(cv);
        col[33 * r] = Y;
    };
#pragma unroll 1
    for (int r0 = 0; r0 < nr4; r0 += 4) {
        double av[4], cv[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) assemble(r0 + t, av[t], cv[t]);
#pragma unroll
        for (int t = 0; t < 4; ++t) advance(r0 + t, av[t], cv[t]);
    }
#pragma unroll 1
    for (int r = nr4; r < nr; ++r) {
        double av, cv;
        assemble(r, av, cv);
        advance(r, av, cv);
    }
    // publish the block's map; clear the slot of the next iteration (its last
    // readers are behind the barrier that started this one)
    const int par = m & 1;
    st_map(map_slot(I, par, blk, vt), not_empty(P), not_empty(fma(-P, X0, Y)));
    {
        const double e = __longlong_as_double((long long)kEmptyBits);
        st_map(map_slot(I, par ^ 1, blk, vt), e, e);
    }
    // previous iterate (f^n at m = 0), streamed 8 rows ahead
    double* pw = fo + g.first;
    double c0[4], c1[4];
    if (kResidual) {
        if (nr4 > 0) ld4(c0, po, st);
        if (nr4 > 4) ld4(c1, po + 4 * st, st);
    }
    double X;
    const bool ok = fold_carry(I, g, fn, par, blk, vt, G, limit, X);
    // rows: x = Y + (a_0 .. a_r) (X - X0).  With non-negative right-hand sides
    // the correction's share only shrinks along the scan (x_r >= a_r x_{r-1}),
    // so once it is below 2^-56 for every lane the remaining rows are exact as
    // they are; a tile with a negative one corrects all its rows.
    const bool keep = __any_sync(0xffffffffu, neg < 0 || !(X >= 0.0));
    double Pc = X - X0;
    bool corr = keep || __any_sync(0xffffffffu, !(fabs(Pc) <= 1.3877787807814457e-17 * X));
    const double tol = I.tol, abs_tol = I.abs_tol;
    const bool strict = !(abs_tol > 1e-290 && tol >= 0.0);
    auto rows4 = [&](int r0, double (&o)[4]) {
        double x[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) x[t] = col[33 * (r0 + t)];
        if (corr) {
            double a[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) a[t] = cpl * recip3(one_plus + co[r0 + t][3]);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                Pc *= a[t];
                x[t] += Pc;
                col[33 * (r0 + t)] = x[t];
            }
            corr = keep || __any_sync(0xffffffffu, !(fabs(Pc) <= 1.3877787807814457e-17 * fabs(x[3])));
        }
        if (kResidual) {
#pragma unroll
            for (int t = 0; t < 4; ++t) residual(x[t], o[t], tol, abs_tol, strict, q1, q2);
        }
        if (g.lane_ok) {
#pragma unroll
            for (int t = 0; t < 4; ++t) pw[t * st] = x[t];
        }
        pw += 4 * st;
    };
    po += 8 * st;
#pragma unroll 1
    for (int r0 = 0; r0 < nr4; r0 += 8) {
        rows4(r0, c0);
        if (kResidual && r0 + 8 < nr4) ld4(c0, po, st);
        if (r0 + 4 < nr4) {
            rows4(r0 + 4, c1);
            if (kResidual && r0 + 12 < nr4) ld4(c1, po + 4 * st, st);
        }
        po += 8 * st;
    }
#pragma unroll 1
    for (int r = nr4; r < nr; ++r) {
        double x = col[33 * r];
        if (corr) {
            Pc *= cpl * recip3(one_plus + co[r][3]);
            x += Pc;
            col[33 * r] = x;
        }
        if (kResidual)
            residual(x, __ldcg((m > 0 ? fo : fn) + g.first + r * st), tol, abs_tol, strict, q1, q2);
        if (g.lane_ok) *pw = x;
        pw += st;
    }
    __syncwarp();
    // a sum that is not finite: some x may not be (or the sum overflowed)
    if (__any_sync(0xffffffffu, !row_sums(w, g, I.rblk, vt, part))) {
        bool nf = false;
        for (int r = 0; r < nr; ++r) nf |= !isfinite(w.a[r][lane]);
        if (nf && g.lane_ok) {
            bad = true;
            // |x - o| / (...) of a non-finite x is NaN, and the maximum propagates it
            q1.special = q2.special = __longlong_as_double(0x7ff8000000000000ll);
        }
    }
    __syncwarp();
    return ok;
}

// Coefficients of row `k` of a block of nr rows into C.coef.
__device__ __forceinline__ void put_coef(CtaSmem& C, int k, int nr, const double* c4) {
    const double2 a = make_double2(c4[0], c4[1]), b = make_double2(c4[2] * c4[3], c4[3]);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        double2* p = reinterpret_cast<double2*>(C.coef[d][d == 0 ? k : nr - 1 - k]);
        p[0] = a;
        p[1] = b;
    }
}

// The same for the rows of a block and for another CTA (HBM).
__device__ __forceinline__ void save_coef(CtaSmem& C, int i, int k, int nr, const double* c4) {
    const ImpInst& I = C.I;
    reinterpret_cast<double2*>(&I.Wc[4 * (size_t)i])[0] = make_double2(c4[0], c4[1]);
    reinterpret_cast<double2*>(&I.Wc[4 * (size_t)i])[1] = make_double2(c4[2], c4[3]);
    put_coef(C, k, nr, c4);
}

// Bound G of the fold for iteration m.  T is at least 1e-12 from the first
// update on, so a Maxwellian is at most 4e5 n (asum: sum of the |weights| of
// an Anderson combination, plus one); the first coefficients (T floored at
// 1e-300) have a maximum of their own.
__device__ __forceinline__ double fold_bound(double fmax_, double cmax0, double nm, int m, double asum) {
    const double mb = m == 0 ? cmax0 : 4.0e5 * nm * asum;
    return fmax_ > mb ? fmax_ : mb;
}

// Anderson-combined W of one row (bgk1d_aa_cpu.py:170-188: floors, |u| <=
// u_max) from the weighted history sums and the newest moments; W and the
// coefficients of the row are stored (lane = row, ok = the row exists).
__device__ __forceinline__ void combine_row(CtaSmem& C, int i, int nr, bool ok, const double* acc,
                                            const double* wnew) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int nx = I.nx;
    double wv[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) wv[q] = acc[q] * I.aa_beta + (1.0 - I.aa_beta) * wnew[q];
    const double n1 = clamp_min_t(wv[0], 1e-12);
    const double Tm = clamp_min_t(wv[2], 1e-12);
    double um = div_nr(wv[1], n1);
    if (!isfinite(um)) um = 0.0;
    um = um < -I.u_max ? -I.u_max : (um > I.u_max ? I.u_max : um);
    const double num = n1 * um;
    double c4[4];
    row_coeffs_nr(I.tau_tilde, I.dt, n1, num, Tm, c4);
    if (ok) {
        I.W[i] = n1;
        I.W[nx + i] = num;
        I.W[2 * nx + i] = Tm;
        put_coef(C, lane, nr, c4);
    }
}

// Row coefficients of W^(m) for the item's rows (warp 0, lane = row) into
// C.coef, and the bound of the fold.  After an applied Anderson call the
// combination is formed here from the history in HBM.
__device__ __noinline__ void stage_rows_coef(CtaSmem& C, int blk, int m, bool cached) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int nx = I.nx, n_inner = I.n_inner;
    const int k0 = blk * I.rblk;
    const int nr = n_inner - k0 < I.rblk ? n_inner - k0 : I.rblk;
    const bool comb = m >= 1 && aa_applies(I, m - 1);
    const double fmx = ld_cg(&I.scal[0]);
    const double cm = ld_cg(&I.scal[1]), nm = ld_cg(&I.scal[2 + m]);
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
        double acc[3], wnew[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            double gv[kMaxAACols];
#pragma unroll
            for (int jj = 0; jj < kMaxAACols; ++jj)
                gv[jj] = ld_cg(&I.aaG[(size_t)col[jj] * d + q * n_inner + kc]);
            wnew[q] = ld_cg(&I.Wn[q * nx + i]);
            acc[q] = 0.0;
#pragma unroll
            for (int jj = 0; jj < kMaxAACols; ++jj) acc[q] = fma(jj < mh ? gv[jj] : 0.0, al[jj], acc[q]);
        }
#pragma unroll
        for (int jj = 0; jj < kMaxAACols; ++jj) asum += jj < mh ? fabs(al[jj]) : 0.0;
        combine_row(C, i, nr, lane < nr, acc, wnew);
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
}

// The combination of a solo plan, by the whole CTA: every CTA sums the Gram
// partials of all blocks and solves the small system itself, which saves the
// round trips of one CTA doing it for all (last-arrival counter, coefficients
// written and read back); the history of the rows is in shared memory.
// Returns the sum of the |weights| plus one (warp 0; others: 1).
__device__ __noinline__ double solo_combine(CtaSmem& C, const Ring& ring, int blk, int m) {
    const ImpInst& I = C.I;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int mh = m < I.aa_cols ? m : I.aa_cols;  // history of call m-1
    const int npairs = mh * (mh + 1) / 2;
    const double* gp = I.gpart + (size_t)((m - 1) & 1) * kMaxPairs * I.nblk;
    for (int t = warp; t < npairs; t += 2 * nw) {
        const int t2 = t + nw < npairs ? t + nw : t;  // two pairs in flight
        double v, v2;
        aa_pair_sum2(gp + (size_t)t * I.nblk, gp + (size_t)t2 * I.nblk, I.nblk, v, v2);
        if (lane == 0) {
            C.gs[t] = v;
            C.gs[t2] = v2;
        }
    }
    __syncthreads();
    double asum = 1.0;
    if (warp == 0) {
        const double al = aa_solve_warp(C.gs, mh, I.aa_reg, I.aa_alpha_max);
        const int k0 = blk * I.rblk;
        const int nr = I.n_inner - k0 < I.rblk ? I.n_inner - k0 : I.rblk;
        const int newest = (m - 1) % I.aa_cols;
        int col = newest + 1 >= mh ? newest + 1 - mh : newest + 1 - mh + I.aa_cols;
        double acc[3] = {0.0, 0.0, 0.0}, wnew[3];
        for (int jj = 0; jj < mh; ++jj) {
            const double aj = __shfl_sync(0xffffffffu, al, jj);
            asum += fabs(aj);
#pragma unroll
            for (int q = 0; q < 3; ++q) acc[q] = fma(ring.G[col][q][lane], aj, acc[q]);
            col = col + 1 == I.aa_cols ? 0 : col + 1;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) wnew[q] = ring.G[newest][q][lane];
        combine_row(C, k0 + lane + 1, nr, lane < nr, acc, wnew);
        if (lane == 0) C.gbound = asum;
    }
    __syncthreads();
    return C.gbound;
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
// residual, Anderson history, W and coefficients of the next
// iteration (keq_implicit.cu reduce_block has the reference lines).  nm:
// largest n of the iterates before.  With `early`, lane 0 makes its half of
// the CTA's arrival at the grid barrier as soon as everything that other CTAs wait for is out (its W and
// coefficients are read by this CTA alone then), so that the rest overlaps the
// barrier.  In an applied Anderson call the older residual columns go to
// w.a[row][3 j + q] unless they are in the ring.
__device__ __noinline__ void finish_item(CtaSmem& C, TileBuf& w, Ring* ring, const double (*part)[3][32],
                                         int blk, int m, double nm, GridBarrier* early) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int k0 = blk * I.rblk, k = k0 + lane;
    const int nr = I.n_inner - k0 < I.rblk ? I.n_inner - k0 : I.rblk;
    const bool ok = lane < nr;
    const int i = k + 1;
    const int nx = I.nx, n_inner = I.n_inner, d = 3 * n_inner;
    const double s0 = slot_sum(part, I.nvt, 0);
    if (m + 1 < I.picard_iter) {  // largest n of the iterates so far (rounded up to its high word)
        const double n1 = s0 * I.dv;
        const unsigned mh = __reduce_max_sync(
            0xffffffffu, ok ? (unsigned)__double2hiint(n1 > 1e-12 ? n1 : 1e-12) : 0u);
        const double mx = __hiloint2double((int)mh, -1);
        if (lane == 0) atomic_max_nonneg(&I.scal[2 + m + 1], mx > nm ? mx : nm);
    }
    if (early != nullptr && lane == 0) bar_arrive_nr(early, 1u);
    const double s1 = slot_sum(part, I.nvt, 1), s2 = slot_sum(part, I.nvt, 2);
    const bool aa_now = aa_applies(I, m);
    const int cols = I.aa_cols > 0 ? I.aa_cols : 1;
    const int head_in = I.aa_on ? m % cols : 0;
    const int mh = (m + 1) < cols ? (m + 1) : cols;
    const bool need_old = I.conv_type == 1 || I.aa_on;
    double wn[3] = {0.0, 0.0, 0.0}, wo[3] = {0.0, 0.0, 0.0}, c4[4];
    if (ok) {
        if (need_old) {
            wo[0] = ld_cg(&I.W[i]);
            wo[1] = ld_cg(&I.W[nx + i]);
            wo[2] = ld_cg(&I.W[2 * nx + i]);
        }
        moments_and_coeffs(s0, s1, s2, I.dv, I.dt, I.tau_tilde, 1e-12, wn, c4);
    }
    if (I.aa_on) {
        if (ring != nullptr) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                ring->G[head_in][q][lane] = wn[q];
                ring->R[head_in][q][lane] = ok ? wn[q] - wo[q] : 0.0;
            }
        } else {
            if (aa_now) {
                int col = head_in + 1 >= mh ? head_in + 1 - mh : head_in + 1 - mh + cols;
                for (int jj = 0; jj < mh - 1; ++jj) {
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        w.a[lane][3 * jj + q] =
                            ok ? ld_cg(&I.aaR[(size_t)col * d + q * n_inner + k]) : 0.0;
                    col = col + 1 == cols ? 0 : col + 1;
                }
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
    }
    if (I.conv_type == 1) {  // bgk1d_conv_util.py:35-58 over all nx cells
        const double at = I.abs_tol, tl = I.tol;
        FracMax q1, q2;
        if (ok) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double df = fabs(wn[q] - wo[q]);
                const double ref = nan_max(fabs(wn[q]), fabs(wo[q]));
                q1.add(df, at + tl * ref);
                q2.add(df, (ref != ref || ref >= at) ? ref : at);
            }
        }
        if (blk == 0 && lane < 2) {  // the two boundary rows
            const int ib = lane == 0 ? 0 : nx - 1;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double a = ld_cg(&I.Wb[3 * lane + q]), o = ld_cg(&I.W[q * nx + ib]);
                const double df = fabs(a - o);
                const double ref = nan_max(fabs(a), fabs(o));
                q1.add(df, at + tl * ref);
                q2.add(df, (ref != ref || ref >= at) ? ref : at);
            }
        }
        const double r1 = warp_max(q1.value()), r2 = warp_max(q2.value());
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

// Gram partials of an applied Anderson call over the block's rows: a warp per
// pair of columns, a lane per row.  After a CTA barrier behind finish_item.
__device__ __forceinline__ void gram_partials(const CtaSmem& C, const TileBuf& w, const Ring* ring,
                                              double* gp, int blk, int m) {
    const ImpInst& I = C.I;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int cols = I.aa_cols;
    const int mh = (m + 1) < cols ? (m + 1) : cols;
    const int newest = m % cols;
    const int col0 = newest + 1 >= mh ? newest + 1 - mh : newest + 1 - mh + cols;
    const int npairs = mh * (mh + 1) / 2;
    for (int t = warp; t < npairs; t += nw) {
        int p = 0, rem = t;
        while (rem >= mh - p) {
            rem -= mh - p;
            ++p;
        }
        const int q = p + rem;
        double v = 0.0;
        if (ring != nullptr) {
            const int cp = col0 + p >= cols ? col0 + p - cols : col0 + p;
            const int cq = col0 + q >= cols ? col0 + q - cols : col0 + q;
#pragma unroll
            for (int c = 0; c < 3; ++c) v = fma(ring->R[cp][c][lane], ring->R[cq][c][lane], v);
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) v = fma(w.a[lane][3 * p + c], w.a[lane][3 * q + c], v);
        }
        v = warp_sum(v);
        if (lane == 0) gp[(size_t)t * I.nblk + blk] = v;
    }
}

// Last block of an instance's Anderson call (warp 0 of its CTA): Gram matrix,
// coefficients into I.alpha.
__device__ __noinline__ void last_block_alpha(CtaSmem& C, int m) {
    const ImpInst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int mh = (m + 1) < I.aa_cols ? (m + 1) : I.aa_cols;
    const int npairs = mh * (mh + 1) / 2;
    for (int t = 0; t < npairs; t += 2) {
        const int t2 = t + 1 < npairs ? t + 1 : t;
        double v, v2;
        aa_pair_sum2(I.gpart + (size_t)t * I.nblk, I.gpart + (size_t)t2 * I.nblk, I.nblk, v, v2);
        if (lane == 0) {
            C.gs[t] = v;
            C.gs[t2] = v2;
        }
    }
    __syncwarp();
    const double al = aa_solve_warp(C.gs, mh, I.aa_reg, I.aa_alpha_max);
    if (lane < mh) I.alpha[(size_t)m * kMaxAACols + lane] = al;
    __syncwarp();
}

// Moments of a boundary row (one warp) into Wb and W, and its copy into f_out.
__device__ __noinline__ double boundary_row(const ImpInst& I, const double* fn, double* fo, int side) {
    const int lane = threadIdx.x & 31;
    const size_t ib = side == 0 ? 0 : (size_t)(I.nx - 1);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, mx = 0.0;
#pragma unroll 4
    for (int j = lane; j < I.nv; j += 32) {
        const double x = __ldcg(&fn[ib * I.nv + j]), v = __ldg(&I.v[j]);
        fo[ib * I.nv + j] = x;
        s0 += x;
        s1 = fma(x, v, s1);
        s2 = fma(x, v * v, s2);
        mx = fabs(x) > mx ? fabs(x) : mx;
    }
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    double n, nu, T;
    moments_from_sums(s0, s1, s2, I.dv, &n, &nu, &T);
    if (lane == 0) {
        I.Wb[3 * side + 0] = n;
        I.Wb[3 * side + 1] = nu;
        I.Wb[3 * side + 2] = T;
        I.W[ib] = n;
        I.W[I.nx + ib] = nu;
        I.W[2 * (size_t)I.nx + ib] = T;
    }
    return mx;
}

// Item of the prologue: moments of f^n, W^(0) and its coefficients, the bounds
// of the fold, empty map slots of both parities.
__device__ __noinline__ void first_item(CtaSmem& C, TileBuf* bufs, double (*part)[3][32], int blk,
                                        const double* __restrict__ fn, double* __restrict__ fo) {
    const ImpInst& I = C.I;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    TileBuf& w = bufs[warp];
    double mx = 0.0;
    for (int vt = warp; vt < I.nvt; vt += nw) {
        const Tile g = make_tile(I, blk, vt);
        copy_tile(I, w, g, fn);
        const double e = __longlong_as_double((long long)kEmptyBits);
        st_map(map_slot(I, 0, blk, vt), e, e);
        st_map(map_slot(I, 1, blk, vt), e, e);
        cp_async_wait_all();
        const double vj = w.vw[lane].x;
        w.vw[lane].y = vj * vj;
        for (int r = 0; r < g.nr; ++r) {
            const double x = fabs(w.a[r][lane]);
            mx = x > mx ? x : mx;
        }
        __syncwarp();
        row_sums(w, g, I.rblk, vt, part);
        __syncwarp();
    }
    if (blk == 0 && warp == nw - 1) {
        const double b = boundary_row(I, fn, fo, 0);
        mx = b > mx ? b : mx;
    }
    if (blk == I.nblk - 1 && warp == nw - 2) {
        const double b = boundary_row(I, fn, fo, 1);
        mx = b > mx ? b : mx;
    }
    mx = warp_max_bits(mx);
    if (lane == 0) C.red[warp][0] = mx;
    __syncthreads();
    if (warp == 0) {
        mx = warp_max_bits(lane < nw ? C.red[lane][0] : 0.0);
        const int k = blk * I.rblk + lane;
        const int nr = I.n_inner - blk * I.rblk < I.rblk ? I.n_inner - blk * I.rblk : I.rblk;
        double n = 0.0, cm = 0.0;
        if (lane < nr) {
            double w3[3], c4[4];
            moments_and_coeffs(slot_sum(part, I.nvt, 0), slot_sum(part, I.nvt, 1),
                               slot_sum(part, I.nvt, 2), I.dv, I.dt, I.tau_tilde, 0.0, w3, c4);
            const int i = k + 1;
            n = w3[0];
            I.W[i] = w3[0];
            I.W[I.nx + i] = w3[1];
            I.W[2 * I.nx + i] = w3[2];
            save_coef(C, i, lane, nr, c4);
            cm = c4[2];
        }
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

__global__ void __launch_bounds__(512, 1)
implicit_rows_kernel(PlanDev* __restrict__ Pp, int swap_io) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
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
    TileBuf* bufs = reinterpret_cast<TileBuf*>(part + nslot);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const bool listed = n_inst > 1 && n_inst <= kListMax;
    int* aoff = reinterpret_cast<int*>(bufs + nw);
    unsigned short* aidx = reinterpret_cast<unsigned short*>(aoff + kListMax + 1);
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
        first_item(C, bufs, part, (int)(t - C.I.item_off), swap_io ? C.I.f_out : C.I.f_in,
                   swap_io ? const_cast<double*>(C.I.f_in) : C.I.f_out);
        coef_item = t;
    }
    // One instance with a CTA for every block: the item, its coefficients, its
    // Anderson history and the next f^n copy stay with the CTA from one
    // iteration to the next.
    const bool solo = n_inst == 1 && total_items <= (long long)G;
    const bool mine = solo && (long long)blockIdx.x < total_items;
    Ring* ring = nullptr;
    if (solo) {
        stage_inst(C, P, 0, cur_b);
        if (mine && warp < C.I.nvt)
            copy_tile(C.I, bufs[warp], make_tile(C.I, (int)blockIdx.x, warp),
                      swap_io ? C.I.f_out : C.I.f_in);
        if (P.ring) ring = reinterpret_cast<Ring*>(aoff);
    }
    bool arrived = false, gave_up = false;
    for (int m = -1; m < max_iter; ++m) {
        // grid barrier that ends iteration m (-1: the prologue)
        if (m >= 0) {
            long long items = total_items;
            double Gb = 0.0, nm = 0.0;
            bool comb = false;
            if (solo) {
                // every thread reads the step's state itself: no CTA barrier
                const ImpInst& I = C.I;
                if (m >= I.picard_iter) break;
                const double fmx = ld_cg(&I.scal[0]), cm = ld_cg(&I.scal[1]);
                nm = ld_cg(&I.scal[2 + m]);
                if (!inst_active_rows(I, m)) break;
                comb = mine && m >= 1 && aa_applies(I, m - 1);
                const double asum = comb ? solo_combine(C, *ring, (int)blockIdx.x, m) : 1.0;
                Gb = fold_bound(fmx, cm, nm, m, asum);
            } else if (listed) {
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
            arrived = false;
            for (long long t = blockIdx.x; t < items;) {
                int blk = (int)t;
                if (!solo) {
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
                }
                const ImpInst& I = C.I;
                const long long item = I.item_off + blk;
                if (solo || listed || inst_active_rows(I, m)) {
                    const double* fn = swap_io ? I.f_out : I.f_in;
                    double* fo = swap_io ? const_cast<double*>(I.f_in) : I.f_out;
                    if (!solo) {
                        if (warp < I.nvt) copy_tile(I, bufs[warp], make_tile(I, blk, warp), fn);
                        if (warp == 0) stage_rows_coef(C, blk, m, coef_item == item);
                        __syncthreads();
                        Gb = C.gbound;
                        nm = C.nm;
                    }
                    FracMax q1, q2;
                    bool bad = false, ok = true;
                    for (int vt = warp; vt < I.nvt; vt += nw) {
                        const Tile g = make_tile(I, blk, vt);
                        ok &= I.conv_type == 0
                                  ? sweep_tile<true>(C, bufs[warp], part, g, blk, vt, m, Gb, limit, fn, fo, q1, q2, bad)
                                  : sweep_tile<false>(C, bufs[warp], part, g, blk, vt, m, Gb, limit, fn, fo, q1, q2, bad);
                        if (vt + nw < I.nvt) copy_tile(I, bufs[warp], make_tile(I, blk, vt + nw), fn);
                    }
                    if (!ok && lane == 0) {
                        atomicOr(&P.head.err, 1 << KEQ_ERR_TIMEOUT);
                        atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
                    }
                    if (I.conv_type == 0) {
                        double r1, r2;
                        frac_values(q1, q2, r1, r2);
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
                    if (!single && threadIdx.x == 64) C.next[claim_par] = G + atomicAdd(&tickets[m], 1u);
                    arrived = solo && !I.aa_on && I.conv_type == 0;
                    if (warp == 0) finish_item(C, bufs[0], ring, part, blk, m, nm, arrived ? bar : nullptr);
                    if (warp == 1) {
                        flush_residuals(C, m);
                        if (arrived && lane == 0) bar_arrive_nr(bar, 1u);
                    }
                    // the next iteration's f^n
                    if (solo && warp < I.nvt) copy_tile(I, bufs[warp], make_tile(I, blk, warp), fn);
                    coef_item = item;
                    if (aa_applies(I, m)) {
                        __syncthreads();
                        gram_partials(C, bufs[0], ring,
                                      I.gpart + (ring ? (size_t)(m & 1) * kMaxPairs * I.nblk : 0), blk, m);
                        if (ring == nullptr) {
                            __syncthreads();
                            if (warp == 0) {
                                unsigned prev = 0;
                                if (lane == 0) {
                                    fence_acq_rel();
                                    prev = atomicAdd(&I.rbdone[m], 1u);
                                    fence_acq_rel();
                                }
                                prev = __shfl_sync(0xffffffffu, prev, 0);
                                if (prev == (unsigned)I.nblk - 1) last_block_alpha(C, m);
                            }
                        }
                    }
                } else if (!single && threadIdx.x == 64) {
                    C.next[claim_par] = G + atomicAdd(&tickets[m], 1u);
                }
                if (single) break;
                __syncthreads();
                t = C.next[claim_par];
                claim_par ^= 1;
            }
            if (traced) trace_mark(P, m, 1, false);
        }
        // two arrivals per CTA; warp 1 waits, while warp 0 may still be busy
        bar_target += 2u * G;
        if (!arrived) __syncthreads();  // uniform in the CTA
        if (threadIdx.x == 32) {
            if (!arrived) bar_arrive_nr(bar, 2u);
            C.ok = bar_wait(bar, bar_target, &P.head.err, limit) ? 1 : 0;
            if (!C.ok) atomicOr(&P.head.err_sticky, 1 << KEQ_ERR_TIMEOUT);
        }
        __syncthreads();
        if (!C.ok) {
            gave_up = true;
            break;
        }
    }
    cp_async_wait_all();
    if (gave_up) return;

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
        keq_step_stats* s = I.stats;
        int aa_applied = 0;
        for (int m = 0; m < last; ++m)
            if (aa_applies(I, m)) ++aa_applied;
        int status = KEQ_OK;
        if (__ldcg(&I.nonfin[last])) status = KEQ_ERR_NONFINITE;
        if (__ldcg(&P.head.err) & (1 << KEQ_ERR_TIMEOUT)) status = KEQ_ERR_TIMEOUT;
        s->status = status;
        s->iters = last + 1;
        s->aa_applied = aa_applied;
        s->lo_iters = 0;
        s->residual = ld_cg(&I.res[2 * last + 1]);
        s->std_residual = ld_cg(&I.res[2 * last]);
        s->lo_residual = 0.0;
        s->std_lo_residual = 0.0;
        s->max_YI = 0.0;
        s->total_iters += last + 1;
        s->total_steps += 1;
    }
}

}  // namespace rows

const void* implicit_rows_entry() { return (const void*)rows::implicit_rows_kernel; }
size_t implicit_rows_smem(int warps, int nslot, int n_inst, int ring) {
    return sizeof(rows::CtaSmem) + (size_t)nslot * 3 * 32 * sizeof(double) + (size_t)warps * sizeof(rows::TileBuf) +
           (n_inst > 1 ? 6 * (rows::kListMax + 2) : 0) + (ring ? sizeof(rows::Ring) : 0);
}

}  // namespace keq
