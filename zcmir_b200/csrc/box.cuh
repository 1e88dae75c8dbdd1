// Summed-area tables of a side's moment planes (box.cu): their layout and a shift's box.
#pragma once

#include <cuda_runtime.h>

namespace zc {

// Comps of a table of nf features: the nf feature sums, then the products in row order, padded to
// whole double2s. Pair q of entry (x, y), the sums over rows ≤ y and columns ≤ x, is the double2 at
// (y·pairs + q)·cw + x: a warp's entries of consecutive columns are consecutive in memory (whole
// entries side by side made each load touch four times the cache lines).
//
// Entries are float64: the four of a box cancel down to its own sum, and rounding that scales with the
// whole plane's sums would be left in it (a 40 × 8 image over one of 360 × 337, whose covariances are near
// singular, had the wrong peak from float32 entries).
__host__ __device__ constexpr int box_comps(int nf) { return nf + nf * (nf + 1) / 2; }
__host__ __device__ constexpr int box_pad(int nf) { return (box_comps(nf) + 1) / 2 * 2; }
// product k of nf features in row order: its two features
__host__ __device__ constexpr int box_i(int k, int nf) {
    int i = 0;
    while (k >= nf - i) k -= nf - i, ++i;
    return i;
}
__host__ __device__ constexpr int box_j(int k, int nf) {
    int i = 0;
    while (k >= nf - i) k -= nf - i, ++i;
    return i + k;
}
// the comp of nf features' product (i, j), i ≤ j
__host__ __device__ constexpr int box_comp(int i, int j, int nf) {
    int k = nf;
    while (!(box_i(k - nf, nf) == i && box_j(k - nf, nf) == j)) ++k;
    return k;
}

// a rectangle of grid cells [x0, x1) × [y0, y1)
struct Box {
    int x0, x1, y0, y1;
};

// The tables the score reads in place of correlations. mode 0: none; 1: side A's moments over side
// B's box (ta, b); 2: also side B's over A's box (tb, a).
struct BoxSums {
    int mode = 0;
    const double *ta = nullptr, *tb = nullptr;
    int cw = 0, ch = 0;
    Box a{}, b{};
};

// A table's sums over the box [x0, x1) × [y0, y1) clipped to the grid, all comps: four corner reads of
// whole entries, of which those on the grid's first row or column are zero and not made. Lanes of
// consecutive shifts read consecutive entries at the corners that move with the shift and one entry
// at those the grid's edge holds. A row's two corners are loaded whole before they are used: taken pair by
// pair, the loads followed one another (score of a 2048² map at a translation 0.44 → 0.31 ms). The
// sums leave as float32, as a transform's do (their own rounding only; float64 ones would not fit the score's
// registers).
template <int NF>
__device__ __forceinline__ void box_read(float (&v)[box_pad(NF)], const double* __restrict__ t, int cw, int ch, int x0,
                                         int x1, int y0, int y1) {
    constexpr int NP = box_pad(NF);
    x0 = max(x0, 0), y0 = max(y0, 0), x1 = min(x1, cw), y1 = min(y1, ch);
#pragma unroll
    for (int i = 0; i < NP; ++i) v[i] = 0.f;
    if (x1 <= x0 || y1 <= y0) return;
    const double2* p = reinterpret_cast<const double2*>(t);
    const size_t r0 = (size_t)(y0 - 1) * (NP / 2) * cw, r1 = (size_t)(y1 - 1) * (NP / 2) * cw;
    const double2 zero = make_double2(0.0, 0.0);
    double d[NP];
    auto row = [&](size_t r, bool sub) {
        double2 hi[NP / 2], lo[NP / 2];
#pragma unroll
        for (int q = 0; q < NP / 2; ++q) {
            hi[q] = __ldg(p + r + (size_t)q * cw + x1 - 1);
            lo[q] = x0 > 0 ? __ldg(p + r + (size_t)q * cw + x0 - 1) : zero;
        }
#pragma unroll
        for (int q = 0; q < NP / 2; ++q) {
            const double a = hi[q].x - lo[q].x, b = hi[q].y - lo[q].y;
            d[2 * q] = sub ? d[2 * q] - a : a;
            d[2 * q + 1] = sub ? d[2 * q + 1] - b : b;
        }
    };
    row(r1, false);
    if (y0 > 0) row(r0, true);
#pragma unroll
    for (int i = 0; i < NP; ++i) v[i] = (float)d[i];
}

}  // namespace zc
