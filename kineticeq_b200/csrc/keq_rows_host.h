// keq_rows_host.h -- host-side choices of the row-block kernels.
#pragma once

#include <math.h>

#include "keq_internal.h"

namespace keq {

// Warps per CTA that suit nvt velocity tiles.
inline int rows_warps(int nvt) { return nvt <= 4 ? 4 : (nvt <= 8 ? 8 : 16); }

// Rows per block: a property of the instance alone, so that its result does not
// depend on the plan it is part of.  The fewest rows (a multiple of 4, at least
// 8, at most 32) that put one block on every CTA of the chip (148 SMs, 16 warps
// each), in as many rounds as 32 rows need.
inline int rows_per_block(int n_inner, int nvt) {
    const int ctas = 148 * (16 / rows_warps(nvt));
    const int rounds = (n_inner + ctas * KEQ_ROWS_MAX - 1) / (ctas * KEQ_ROWS_MAX);
    int r = (n_inner + ctas * rounds - 1) / (ctas * rounds);
    r = (r + 3) / 4 * 4;
    return r < 8 ? 8 : (r > KEQ_ROWS_MAX ? KEQ_ROWS_MAX : r);
}

// Blocks that a carry is folded over at most: with a <= c / (1 + c), c the
// largest coupling, the product over that many blocks is below 2^-200
// (139 > 200 ln 2).
inline int rows_kmax(double c, int rblk) {
    const double la = log1p(1.0 / c);  // -ln(c / (1 + c))
    const double k = 139.0 / (la * rblk);
    return k < 1e6 ? (int)k + 2 : 1000000;
}
constexpr int kRowsKmax = 64;  // a row-block kernel takes an instance up to here

}  // namespace keq
