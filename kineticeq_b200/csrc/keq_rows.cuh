// keq_rows.cuh -- sweep of one velocity tile over one row block, shared by the
// row-block kernels: keq_implicit_solo.cu (one instance, one CTA per block),
// keq_implicit_rows.cu (any plan) and keq_holo_rows.cu (HOLO).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "keq_common.cuh"
#include "keq_implicit.cuh"
#include "keq_internal.h"
#include "keq_tile.cuh"

namespace keq {
namespace rows {

constexpr int kRows = KEQ_ROWS_MAX;
constexpr int kFold = 4;       // maps that a fold loads at a time
constexpr int kSlots = 16;  // partial-sum slots: v-tile vt adds into slot vt & 15

struct TileBuf {
    double2 vw[32];       // (v, v^2) of the tile's lanes
    double a[kRows][33];  // f^n, then Y of the zero-inflow recurrence, then x, in scan order
};
// Bytes of a tile buffer that holds up to `rows` rows.
__host__ __device__ constexpr size_t buf_bytes(int rows) {
    return (offsetof(TileBuf, a) + (size_t)rows * 33 * sizeof(double) + 15) / 16 * 16;
}

// The part of a CTA's shared memory that a sweep reads (Inst: the instance
// record, implicit or HOLO).
template <class Inst>
struct alignas(16) BlockSmemT {
    Inst I;
    // u, -1/(2T), dt/tau n/sqrt(2 pi T), dt/tau per row, in both scan orders
    alignas(16) double coef[2][kRows][4];
};

using BlockSmem = BlockSmemT<ImpInst>;

// read as double2
static_assert(offsetof(BlockSmem, coef) % 16 == 0 && sizeof(BlockSmem) % 16 == 0, "alignment");
static_assert(offsetof(TileBuf, vw) % 16 == 0 && sizeof(TileBuf) % 16 == 0, "alignment");

// e^x for x <= 0 as exp_nonpos (keq_common.cuh), with results below 2^-1021
// flushed to zero and the scale 2^k added to the exponent field, which saves
// two FP64 operations and the compare of the clamp.  e^r = 1 + r + r^2 q(r) with
// q of degree 9, fitted by a Remez exchange for the relative error of e^r on
// |r| <= ln 2 / 2 with the leading coefficient fixed at a double (3.9e-18 with
// the others rounded; the Taylor polynomial of degree 13 has 4.1e-18).  The even
// and odd halves of q side by side make the chain 8 operations instead of 13.
// A NaN does not come out as one: see amplitude().
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
    const double r2 = r * r;
    double e = 2.76307620969295e-07, o = 2.5020624775339694e-08;
    e = fma(e, r2, 2.480149173347253e-05);
    o = fma(o, r2, 2.755752931497712e-06);
    e = fma(e, r2, 0.001388888894486843);
    o = fma(o, r2, 0.0001984126956142306);
    e = fma(e, r2, 0.041666666666525784);
    o = fma(o, r2, 0.008333333333473403);
    e = fma(e, r2, 0.5000000000000011);
    o = fma(o, r2, 0.16666666666666438);
    double p = fma(o, r, e);
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

template <class Inst>
__device__ __forceinline__ Tile make_tile(const Inst& I, int blk, int vt) {
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

// Exchange of the blocks' maps (P, Y) for kernels whose iterations are
// separated by grid barriers: one 16-byte record per lane, empty (a NaN that no
// arithmetic makes) until it is published, two sets by iteration parity.
struct BarrierMaps {
    static constexpr unsigned long long kEmptyBits = ~0ull;
    static __device__ __forceinline__ double2* slot(const ImpInst& I, int par, int blk, int vt) {
        return I.xch + (((size_t)par * I.nblk + blk) * I.nvt + vt) * 32 + (threadIdx.x & 31);
    }
    static __device__ __forceinline__ bool is_empty(double v) {
        return (unsigned long long)__double_as_longlong(v) == kEmptyBits;
    }
    static __device__ __forceinline__ void st(double2* p, double x, double y) {
        asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(x), "d"(y) : "memory");
    }
    static __device__ __forceinline__ void clear(double2* p) {
        const double e = __longlong_as_double((long long)kEmptyBits);
        st(p, e, e);
    }
    const double2* base;
    long long step;
    __device__ __forceinline__ void publish(const ImpInst& I, int m, int blk, int vt, bool pos, double P,
                                            double Y) {
        // a value that happens to carry the empty pattern goes out as another NaN
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        double2* p = slot(I, m & 1, blk, vt);
        st(p, is_empty(P) ? nan : P, is_empty(Y) ? nan : Y);
        // the slot of the next iteration: its last readers are behind the
        // barrier that started this one
        clear(slot(I, (m & 1) ^ 1, blk, vt));
        base = p;
        step = (long long)(pos ? -1 : 1) * I.nvt * 32;
    }
    // The map k blocks upstream; false while it is not there.
    __device__ __forceinline__ bool get(int k, double& P, double& Y) const {
        asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];"
                     : "=d"(P), "=d"(Y) : "l"(base + k * step) : "memory");
        return !(is_empty(P) || is_empty(Y));
    }
};

// The same for a kernel without barriers: every 64-bit word carries 32 bits of
// a value and a 32-bit tag (the iteration), so a word is valid by itself and
// nothing has to be cleared or ordered.  Two sets by iteration parity, or one
// (both pointers alike) where a block publishes only once it knows that all
// blocks are done with the maps before.
__device__ __forceinline__ void st_tagged(ulonglong2* p, double v, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p),
                 "l"(t | (unsigned)__double2hiint(v)), "l"(t | (unsigned)__double2loint(v)) : "memory");
}
__device__ __forceinline__ bool ld_tagged(const ulonglong2* p, unsigned tag, double& v) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    v = __hiloint2double((int)(unsigned)a, (int)(unsigned)b);
    return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}

// Kernels whose launches the host clears nothing for (a memset in front of every
// launch costs 1.6 to 2 us): every CTA arrives at the launch's one barrier once,
// whatever happens to the launch, so that arrivals / G counts the launches, and
// maxima over the blocks alternate between two sets, of which a launch clears the
// one it does not use.  launch_parity: before the CTA's own arrival.
__device__ __forceinline__ int launch_parity(const unsigned long long* arrivals, unsigned G) {
    unsigned long long n;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(n) : "l"(arrivals) : "memory");
    return (int)(n / G & 1ull);
}
__device__ __forceinline__ bool launch_barrier(unsigned long long* arrivals, unsigned G,
                                               unsigned long long limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long old, now;
        asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;"
                     : "=l"(old) : "l"(arrivals), "l"(1ull) : "memory");
        const unsigned long long target = (old / G + 1ull) * G;
        unsigned long long it = 0;
        unsigned ns = 0;
        s_ok = 1;
        for (;;) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(arrivals) : "memory");
            if (now >= target) break;
            if (++it > limit) {
                s_ok = 0;
                break;
            }
            if (ns) __nanosleep(ns);
            ns = ns ? (ns < 128 ? 2 * ns : ns) : 16;
        }
        fence_acq_rel();
    }
    __syncthreads();
    return s_ok != 0;
}

struct TaggedMaps {
    ulonglong2* maps[2];  // by parity: [block][v-tile][P | Y][lane]
    unsigned tag;
    const ulonglong2* base;
    long long step;
    template <class Inst>
    __device__ __forceinline__ ulonglong2* slot(const Inst& I, int par, int blk, int vt) const {
        return (par ? maps[1] : maps[0]) + ((size_t)blk * I.nvt + vt) * 64 + (threadIdx.x & 31);
    }
    template <class Inst>
    __device__ __forceinline__ void publish(const Inst& I, int m, int blk, int vt, bool pos, double P,
                                            double Y) {
        ulonglong2* p = slot(I, m & 1, blk, vt);
        st_tagged(p, P, tag);
        st_tagged(p + 32, Y, tag);
        base = p;
        step = (long long)(pos ? -1 : 1) * I.nvt * 64;
    }
    __device__ __forceinline__ bool get(int k, double& P, double& Y) const {
        const ulonglong2* p = base + k * step;
        const bool a = ld_tagged(p, tag, P), b = ld_tagged(p + 32, tag, Y);
        return a && b;
    }
};

// Start the copy of the tile's f^n (scan order) and velocities into shared
// memory; lane copies its own column.
template <class Inst>
__device__ __forceinline__ void copy_tile(const Inst& I, TileBuf& w, const Tile& g,
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
// the fold ends when, for every lane, that is below 2^-58 of |X| or 2^-1000 of G
// (where nothing flows in), or after kmax blocks.  The end is relative to X, not
// to a tolerance of the iteration: the far tails of a distribution, 1e-40 and
// less, keep their digits (a bound of 2^-58 of the absolute tolerance 1e-16 left
// 1e-8 to 1 of them, and saved at most one block in seven).  The number of
// blocks folded depends on the data alone, so the result does not depend on
// timing.  An infinite G bounds nothing: all kmax blocks are folded.  False if a
// wait gave up.
template <class Inst, class Maps>
__device__ __forceinline__ bool fold_carry(const Inst& I, const Tile& g, const double* fn,
                                           const Maps& maps, int blk, double G,
                                           unsigned long long limit, double& X) {
    const bool bounded = G <= 1.7976931348623157e308;
    const double eps = bounded ? 3.469446951953614e-18 : 0.0;            // 2^-58
    const double floor_g = bounded ? G * 9.332636185032189e-302 : 0.0;   // 2^-1000
    const int avail = g.pos ? blk : I.nblk - 1 - blk;                    // blocks upstream
    const int last = avail < I.kmax ? avail : I.kmax;
    double acc = 0.0, pr = 1.0;
    for (int k = 1; k <= last; k += kFold) {
        // kFold blocks in flight together (past the last one: the last again)
        double vp[kFold], vy[kFold];
        unsigned long long it = 0;
        for (;;) {
            bool miss = false;
#pragma unroll
            for (int t = 0; t < kFold; ++t) {
                miss |= !maps.get(k + t < last ? k + t : last, vp[t], vy[t]);
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
                acc = fma(pr, vy[t], acc);
                pr *= vp[t];
                const double th = eps * fabs(acc) > floor_g ? eps * fabs(acc) : floor_g;
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

// Sums over the tile's velocities of x (1, v, v^2[, v^3]) per row, added to
// (first tile of the slot: stored into) p.  Lane = row; with 8 or 16 rows the
// columns are split over 4 or 2 lanes per row and combined by shuffles.  Four
// running sums per quantity (columns j, j+1, j+2, j+3 of every four): a single
// one would wait for 32 dependent additions.  Returns whether the lane's sum of
// x is finite.
template <int NQ>
__device__ __forceinline__ bool row_sums(const TileBuf& w, const Tile& g, int rblk, bool first,
                                         double (*p)[32]) {
    const int lane = threadIdx.x & 31;
    const int w2 = rblk <= 8 ? 8 : (rblk <= 16 ? 16 : 32);  // lanes per column group
    const int r = lane & (w2 - 1), grp = lane / w2;
    const int per = w2;  // 32 / (32 / w2) columns per group
    int j = grp * per, je = j + per;
    j = j > g.lo ? j : g.lo;
    je = je < g.hi ? je : g.hi;
    double q[NQ][4];
#pragma unroll
    for (int t = 0; t < NQ; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) q[t][c] = 0.0;
    auto add = [&](double x, double2 vv, int c) {
        q[0][c] += x;
        q[1][c] = fma(x, vv.x, q[1][c]);
        if (NQ == 3) {
            q[2][c] = fma(x, vv.y, q[2][c]);
        } else {
            const double t = x * vv.y;
            q[2][c] += t;
            q[NQ - 1][c] = fma(t, vv.x, q[NQ - 1][c]);
        }
    };
    if (r < g.nr) {
        const double* a = w.a[g.pos ? r : g.nr - 1 - r];
#pragma unroll 2
        for (; j + 4 <= je; j += 4) {
#pragma unroll
            for (int c = 0; c < 4; ++c) add(a[j + c], w.vw[j + c], c);
        }
        for (; j < je; ++j) add(a[j], w.vw[j], 0);
    }
    double s[NQ];
#pragma unroll
    for (int t = 0; t < NQ; ++t) s[t] = (q[t][0] + q[t][1]) + (q[t][2] + q[t][3]);
    for (int o = w2; o < 32; o <<= 1) {
#pragma unroll
        for (int t = 0; t < NQ; ++t) s[t] += __shfl_xor_sync(0xffffffffu, s[t], o);
    }
    if (lane < w2) {
#pragma unroll
        for (int t = 0; t < NQ; ++t) p[t][r] = first ? s[t] : s[t] + p[t][r];
    }
    return isfinite(s[0]);
}

// Row sum of quantity q over nt tiles from their slots (lane = row), in four
// running sums.  All loads are issued together (unused slots repeat the last
// one and are selected out): one warp runs this with its CTA waiting, and as a
// loop three sums took 1300 (4 slots) to 2500 cycles (16).
template <int NQ, int S = kSlots>
__device__ __forceinline__ double slot_sum(const double (*part)[NQ][32], int nt, int q) {
    const int lane = threadIdx.x & 31;
    const int ns = nt < S ? nt : S;
    double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int h = 0; h < S; h += 8) {
        if (h < ns) {
            double v[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) v[t] = part[h + t < ns ? h + t : ns - 1][q][lane];
#pragma unroll
            for (int t = 0; t < 8; ++t) a[t & 3] += h + t < ns ? v[t] : 0.0;
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

// ---- one sweep of one tile ---------------------------------------------------
// Residuals of the implicit step: |x - o| / (abs_tol + tol ref) and |x - o| /
// max(ref, abs_tol), ref = max(|x|, |o|).  With abs_tol > 0 and finite x the
// denominators are positive; otherwise (`strict`) the general update is taken.
// Non-finite x are found from the row sums.
//
// A running maximum of fractions is a chain of 70 cycles per row (two products,
// a compare, two selects); four rows at a time are compared in pairs first, so
// that the running maximum takes one link per four rows.
__device__ __forceinline__ void larger(double& n, double& d, double n1, double d1) {
    const bool t = n1 * d > n * d1;
    n = t ? n1 : n;
    d = t ? d1 : d;
}
struct PicardResidual {
    FracMax q1, q2;
    double tol, abs_tol;
    bool strict;
    __device__ __forceinline__ PicardResidual(double t, double a)
        : tol(t), abs_tol(a), strict(!(a > 1e-290 && t >= 0.0)) {}
    __device__ __forceinline__ void add(double x, double o) {
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
    __device__ __forceinline__ void add4(const double (&x)[4], const double (&o)[4]) {
        if (strict) {
#pragma unroll
            for (int t = 0; t < 4; ++t) add(x[t], o[t]);
            return;
        }
        double n1[4], n2[4], d1[4], d2[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const double ref = fabs(x[t]) > fabs(o[t]) ? fabs(x[t]) : fabs(o[t]);
            n1[t] = n2[t] = fabs(x[t] - o[t]);
            d1[t] = fma(tol, ref, abs_tol);
            d2[t] = ref > abs_tol ? ref : abs_tol;
        }
        larger(n1[0], d1[0], n1[1], d1[1]);
        larger(n1[2], d1[2], n1[3], d1[3]);
        larger(n2[0], d2[0], n2[1], d2[1]);
        larger(n2[2], d2[2], n2[3], d2[3]);
        larger(n1[0], d1[0], n1[2], d1[2]);
        larger(n2[0], d2[0], n2[2], d2[2]);
        larger(q1.num, q1.den, n1[0], d1[0]);
        larger(q2.num, q2.den, n2[0], d2[0]);
    }
    // |x - o| / (...) of a non-finite x is NaN, and the maximum propagates it
    __device__ __forceinline__ void set_nan() {
        q1.special = q2.special = __longlong_as_double(0x7ff8000000000000ll);
    }
    // Values of both maxima, the two quotients interleaved.
    __device__ __forceinline__ void values(double& v1, double& v2) const {
        if (q1.den >= 1e-270 && q1.den <= 1e270 && q2.den >= 1e-270 && q2.den <= 1e270) {
            const double r1 = recip3(q1.den), r2 = recip3(q2.den);
            v1 = refined(q1.num * r1, q1.den, q1.num, r1);
            v2 = refined(q2.num * r2, q2.den, q2.num, r2);
        } else {
            v1 = q1.num / q1.den;
            v2 = q2.num / q2.den;
        }
        // a quotient met on the general path (NaN wins)
        v1 = v1 > q1.special ? v1 : q1.special;
        v2 = v2 > q2.special ? v2 : q2.special;
    }
};

// The tile's right-hand side (f^n; HOLO: the explicit term) is in, or on its
// way to, w.a.  m: iteration (0: the previous iterate is fn, later fo); cscale:
// v to the coupling.
//
// What bounds a sweep (4096x512, 28 rows, 16 warps per CTA, 28000 cycles an
// iteration): the FP64 pipe in the first half (9400 cycles, 80% of the pipe);
// dependent arithmetic with four warps per scheduler in the rows of the second
// (7500 cycles; holding the iterate in shared memory instead of reading and
// writing it took only 600 off); the inflow (2000), the row sums (2300) and the
// row update with the exchange between blocks (5000) are latencies.
//
// First half of a sweep: assembly, the recurrence from the previous iterate's
// inflow, the block's map.  Needs the block's own coefficients only and writes
// nothing but the map.
template <class Maps>
struct SweepState {
    Maps maps;
    double X0;  // inflow that the recurrence started from
    int neg;    // sign bit: a term of the recurrence was negative
};
template <class Inst, class Maps>
__device__ __forceinline__ void sweep_begin(const BlockSmemT<Inst>& C, TileBuf& w, const Tile& g, int blk,
                                            int vt, int m, double cscale, const double* __restrict__ fn,
                                            SweepState<Maps>& S) {
    const Inst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int nr = g.nr, nr4 = nr & ~3;
    const double(*co)[4] = C.coef[g.pos ? 0 : 1];
    double* col = &w.a[0][lane];
    cp_async_wait_all();
    const double vj = w.vw[lane].x;
    w.vw[lane].y = vj * vj;
    const double cpl = cscale * fabs(vj);
    const double one_plus = 1.0 + cpl;
    // The recurrence starts from the previous iterate's inflow X0 instead of
    // zero, so that what is left to correct, the product of the a times
    // (X - X0), dies out sooner (the iterates converge).
    const double X0 = m > 0 ? __ldcg(I.xin + ((size_t)blk * I.nvt + vt) * 32 + lane) : __ldcg(fn + g.first - g.st);
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
    S.maps.publish(I, m, blk, vt, g.pos, P, fma(-P, X0, Y));  // of the zero-inflow recurrence
    S.X0 = X0;
    S.neg = neg;
}

// A block upstream has a row that is NaN (its moments are, so all its velocities
// are).  The fold ends before it gets to blocks far away, where a NaN counts all the
// same.  Either between the halves of a sweep (the correction of every row becomes
// NaN), or before it, by one thread, for the tiles of one direction (0: v > 0): the
// first row's right-hand side becomes NaN.
template <class Maps>
__device__ __forceinline__ void nan_inflow(SweepState<Maps>& S) {
    S.X0 = __longlong_as_double(0x7ff8000000000000ll);
}
template <class Inst>
__device__ __forceinline__ void nan_inflow(BlockSmemT<Inst>& C, int direction) {
    C.coef[direction][0][2] = __longlong_as_double(0x7ff8000000000000ll);
}

// Flags of a block's sweep: non-finite values; a wait gave up, so the block's rows
// are wrong and no block may go on, or end the step, with its record; rows that the
// next sweep makes NaN.
constexpr int kBadValue = 1, kBadWait = 2, kBadNan = 4;

// Second half: inflow, correction of the rows, residual, row sums into the
// tile's partial-sum slot p.
template <bool kResidual, int NQ, class Inst, class Maps, class Res>
__device__ __forceinline__ bool sweep_end(const BlockSmemT<Inst>& C, TileBuf& w, double (*p)[32],
                                          bool first, const Tile& g, int blk, int vt, int m,
                                          double cscale, double G, const SweepState<Maps>& S,
                                          unsigned long long limit, const double* __restrict__ fn,
                                          double* __restrict__ fo, Res& res, bool& bad) {
    const Inst& I = C.I;
    const int lane = threadIdx.x & 31;
    const int nr = g.nr, nr4 = nr & ~3;
    const double(*co)[4] = C.coef[g.pos ? 0 : 1];
    double* col = &w.a[0][lane];
    const double cpl = cscale * fabs(w.vw[lane].x);
    const double one_plus = 1.0 + cpl;
    const long long st = g.st;
    const double* po = (m > 0 ? fo : fn) + g.first;
    double* xin = I.xin + ((size_t)blk * I.nvt + vt) * 32 + lane;
    const double X0 = S.X0;
    const int neg = S.neg;
    // previous iterate (f^n at m = 0), streamed 8 rows ahead
    double* pw = fo + g.first;
    double c0[4], c1[4];
    if (kResidual) {
        if (nr4 > 0) ld4(c0, po, st);
        if (nr4 > 4) ld4(c1, po + 4 * st, st);
    }
    double X;
    const bool ok = fold_carry(I, g, fn, S.maps, blk, G, limit, X);
    __stcg(xin, X);
    // rows: x = Y + (a_0 .. a_r) (X - X0).  With non-negative right-hand sides
    // the correction's share only shrinks along the scan (x_r >= a_r x_{r-1}),
    // so once it is below 2^-56 for every lane the remaining rows are exact as
    // they are; a tile with a negative one corrects all its rows.
    const bool keep = __any_sync(0xffffffffu, neg < 0 || !(X >= 0.0));
    double Pc = X - X0;
    bool corr = keep || __any_sync(0xffffffffu, !(fabs(Pc) <= 1.3877787807814457e-17 * X));
    // The correction first, as far as it is visible, then residuals and stores
    // without votes or branches between the rows.
#pragma unroll 1
    for (int r0 = 0; corr && r0 < nr; r0 += 4) {
        double a[4], x[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int r = r0 + t < nr ? r0 + t : nr - 1;
            x[t] = col[33 * r];
            a[t] = cpl * recip3(one_plus + co[r][3]);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            Pc *= a[t];
            x[t] += Pc;
            if (r0 + t < nr) col[33 * (r0 + t)] = x[t];
        }
        corr = keep || __any_sync(0xffffffffu, !(fabs(Pc) <= 1.3877787807814457e-17 * fabs(x[3])));
    }
    auto rows4 = [&](int r0, double (&o)[4]) {
        double x[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) x[t] = col[33 * (r0 + t)];
        if (kResidual) res.add4(x, o);
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
        const double x = col[33 * r];
        if (kResidual)
            res.add(x, __ldcg((m > 0 ? fo : fn) + g.first + r * st));
        if (g.lane_ok) *pw = x;
        pw += st;
    }
    __syncwarp();
    // a sum that is not finite: some x may not be (or the sum overflowed)
    if (__any_sync(0xffffffffu, !row_sums<NQ>(w, g, I.rblk, first, p))) {
        bool nf = false;
        for (int r = 0; r < nr; ++r) nf |= !isfinite(w.a[r][lane]);
        if (nf && g.lane_ok) {
            bad = true;
            res.set_nan();
        }
    }
    __syncwarp();
    return ok;
}

// Both halves.
template <bool kResidual, int NQ, class Inst, class Maps, class Res>
__device__ __forceinline__ bool sweep_tile(const BlockSmemT<Inst>& C, TileBuf& w, double (*p)[32],
                                           bool first, const Tile& g, int blk, int vt, int m,
                                           double cscale, double G, const Maps& maps,
                                           unsigned long long limit, const double* __restrict__ fn,
                                           double* __restrict__ fo, Res& res, bool& bad) {
    SweepState<Maps> S;
    S.maps = maps;
    sweep_begin(C, w, g, blk, vt, m, cscale, fn, S);
    return sweep_end<kResidual, NQ>(C, w, p, first, g, blk, vt, m, cscale, G, S, limit, fn, fo, res, bad);
}

// The Maxwellian's amplitude, NaN where its argument is: exp_neg does not carry a
// NaN, and a row that overflowed has to stay NaN.
__device__ __forceinline__ double amplitude(const double* c4) {
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    return c4[0] != c4[0] || c4[1] != c4[1] ? nan : c4[2];
}

// Some row of the block has moments that make its next sweep NaN whatever flows in:
// n is NaN or +inf, and with it u (warp, lane = row; n before it is clamped).
__device__ __forceinline__ bool any_nan_row(bool ok, double n) {
    return __any_sync(0xffffffffu, ok && !(n <= 1.7976931348623157e308));
}

// Coefficients of row `k` of a block of nr rows into C.coef.
template <class Smem>
__device__ __forceinline__ void put_coef(Smem& C, int k, int nr, const double* c4) {
    const double2 a = make_double2(c4[0], c4[1]), b = make_double2(amplitude(c4) * c4[3], c4[3]);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        double2* p = reinterpret_cast<double2*>(C.coef[d][d == 0 ? k : nr - 1 - k]);
        p[0] = a;
        p[1] = b;
    }
}

// Largest n of the rows, rounded up to its high word (warp).
__device__ __forceinline__ double n_bound(bool ok, double n) {
    const unsigned h = __reduce_max_sync(0xffffffffu,
                                         ok ? (unsigned)__double2hiint(n > 1e-12 ? n : 1e-12) : 0u);
    return __hiloint2double((int)h, -1);
}

// Bound G of the fold for iteration m.  T is at least 1e-12 from the first
// update on, so a Maxwellian is at most 4e5 n (asum: sum of the |weights| of
// an Anderson combination, plus one); the first coefficients (T floored at
// 1e-300) have a maximum of their own.
__device__ __forceinline__ double fold_bound(double fmax_, double cmax0, double nm, int m, double asum) {
    const double mb = m == 0 ? cmax0 : 4.0e5 * nm * asum;
    return fmax_ > mb ? fmax_ : mb;
}

// Moments of a boundary row (one warp) into Wb and W, and its copy into f_out.
static __device__ __noinline__ double boundary_row(const ImpInst& I, const double* fn, double* fo, int side) {
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

// Anderson-combined W of one row (bgk1d_aa_cpu.py:170-188: floors, |u| <=
// u_max) from the weighted history sums and the newest moments, and the
// coefficients of the row.
__device__ __forceinline__ void combine_row(const ImpInst& I, const double* acc, const double* wnew,
                                            double* w3, double* c4) {
    double wv[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) wv[q] = acc[q] * I.aa_beta + (1.0 - I.aa_beta) * wnew[q];
    const double n1 = clamp_min_t(wv[0], 1e-12);
    const double Tm = clamp_min_t(wv[2], 1e-12);
    double um = div_nr(wv[1], n1);
    if (!isfinite(um)) um = 0.0;
    um = um < -I.u_max ? -I.u_max : (um > I.u_max ? I.u_max : um);
    w3[0] = n1;
    w3[1] = n1 * um;
    w3[2] = Tm;
    row_coeffs_nr(I.tau_tilde, I.dt, w3[0], w3[1], w3[2], c4);
}

// "w" residual of one row, bgk1d_conv_util.py:35-58.
__device__ __forceinline__ void residual_w(const double* wn, const double* wo, double at, double tl,
                                           FracMax& q1, FracMax& q2) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double df = fabs(wn[q] - wo[q]);
        const double ref = nan_max(fabs(wn[q]), fabs(wo[q]));
        q1.add(df, at + tl * ref);
        q2.add(df, (ref != ref || ref >= at) ? ref : at);
    }
}

// FracMax::value with the short division.
__device__ __forceinline__ double frac_value(const FracMax& f) {
    const double q = div_nr(f.num, f.den);
    if (f.special != f.special) return f.special;
    return q > f.special ? q : f.special;
}

// Moments of f^n of a block into the partial-sum slots (all warps), its
// boundary rows; the lane's largest |f^n|.  w: the warp's buffer.
__device__ __forceinline__ double first_tiles(const BlockSmem& C, TileBuf& w, double (*part)[3][32],
                                              int blk, const double* __restrict__ fn,
                                              double* __restrict__ fo, int smask = kSlots - 1) {
    const ImpInst& I = C.I;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    double mx = 0.0;
    for (int vt = warp; vt < I.nvt; vt += nw) {
        const Tile g = make_tile(I, blk, vt);
        copy_tile(I, w, g, fn);
        cp_async_wait_all();
        const double vj = w.vw[lane].x;
        w.vw[lane].y = vj * vj;
        for (int r = 0; r < g.nr; ++r) {
            const double x = fabs(w.a[r][lane]);
            mx = x > mx ? x : mx;
        }
        __syncwarp();
        row_sums<3>(w, g, I.rblk, vt <= smask, part[vt & smask]);
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
    return mx;
}

// Statistics of a step whose last iteration is `last` (one thread).
__device__ __forceinline__ void write_stats(const ImpInst& I, int last, int status, double std_res,
                                            double res) {
    keq_step_stats* s = I.stats;
    int aa_applied = 0;
    for (int m = 0; m < last; ++m)
        if (aa_applies(I, m)) ++aa_applied;
    s->status = status;
    s->iters = last + 1;
    s->aa_applied = aa_applied;
    s->lo_iters = 0;
    s->residual = res;
    s->std_residual = std_res;
    s->lo_residual = 0.0;
    s->std_lo_residual = 0.0;
    s->max_YI = 0.0;
    s->total_iters += last + 1;
    s->total_steps += 1;
}

}  // namespace rows
}  // namespace keq
