// keq_rows_host.h -- host-side choices of the row-block kernels.
#pragma once

#include <math.h>

#include "keq_internal.h"

namespace keq {

// Warps per CTA that suit nvt velocity tiles.
inline int rows_warps(int nvt) { return nvt <= 4 ? 4 : (nvt <= 8 ? 8 : 16); }

// Rows per block: a property of the instance alone, so that its result does not
// depend on the plan it is part of.  The fewest rows (a multiple of 4, at least
// 8, at most 32) that put at most one block on each of the 148 SMs, or as many
// rounds of 148 as 32 rows need.  A second small CTA on an SM shares its FP64
// pipe and adds blocks to every exchange; a larger block adds rows to the chain
// of one sweep.  Measured, us per step: 2000x256 8 rows 138, 16 rows 105, 24 rows
// 111; 3000x256 214, 152, 115 (32 rows: 124); 4096x64 134, 115, 118 (112); below
// one block per SM fewer rows win: 512x256 8 rows 61, 16 rows 68.
// These are single instances.  In a batch, where other instances fill the SMs, tall
// blocks are cheaper a row (keq_implicit_rows.cu): ms per step of 256 instances
// 6.10 by this rule, 4.99 with the rows of the autotuner's table; of 64 instances 1.79
// with either.
inline int rows_per_block(int n_inner) {
    constexpr int kSms = 148;
    const int rounds = (n_inner + kSms * KEQ_ROWS_MAX - 1) / (kSms * KEQ_ROWS_MAX);
    int r = (n_inner + kSms * rounds - 1) / (kSms * rounds);
    r = (r + 3) / 4 * 4;
    return r < 8 ? 8 : (r > KEQ_ROWS_MAX ? KEQ_ROWS_MAX : r);
}

// Blocks behind which a product of couplings a <= c / (1 + c), c the largest one,
// is below 2^-bits.
inline int rows_kmax(double c, int rblk, double bits) {
    const double la = log1p(1.0 / c);  // -ln(c / (1 + c))
    const double k = bits * 0.6931471805599453 / (la * rblk);
    return k < 1e6 ? (int)k + 2 : 1000000;
}
// Instances are admitted to the row-block kernels by the blocks behind which a
// carry has decayed through kAdmitBits; a fold goes on to kFoldBits where the
// tails of a distribution need it (fold_carry).
constexpr double kAdmitBits = 200.0, kFoldBits = 1000.0;
constexpr int kAheadTiles = 8;  // solo kernel: velocity tiles (and warps) up to which it sweeps ahead
constexpr int kRowsKmax = 64;  // a row-block kernel takes an instance up to here

// Progress of a row-block kernel whose blocks outnumber its `grid` resident CTAs.
// Blocks are claimed in order and a warp publishes its next tile's maps once the
// fold of its current one is done, so with T tiles a warp the unclaimed blocks hold
// up at most (T + 1) kmax claimed ones (kmax: blocks that a fold waits for); the
// rest of the CTAs go on.
inline bool rows_progress(int kmax, int nvt, int warps, int grid) {
    return (long long)kmax * ((nvt + warps - 1) / warps + 1) < grid;
}
// Largest kmax for which plans of every size go on, on a device of `sms` SMs: they
// run CTAs of 8 warps, two on an SM, or of 4 warps, at least four on an SM with up
// to twice the tiles a warp.
inline int rows_fold_limit(int nvt, int sms) { return (2 * sms - 1) / ((nvt + 7) / 8 + 1); }
// An instance that the row-block kernels take, by kmax for kAdmitBits (c up to about
// 3 with 8 rows a block, 14 with 32).
inline bool rows_eligible(int kmax, int nvt, int sms) {
    return kmax <= kRowsKmax && kmax <= rows_fold_limit(nvt, sms);
}

}  // namespace keq
