// Summed-area tables of a side's moment planes (box.cu): their layout and a shift's box.
#pragma once

#include <cuda_runtime.h>

namespace zc {

// Comps of a table of nf features: the nf feature sums, then the products in row order, padded to
// whole float4s. Quad q of entry (x, y), the sums over rows ≤ y and columns ≤ x, is the float4 at
// (y·quads + q)·cw + x: a warp's entries of consecutive columns are consecutive in memory (whole
// entries side by side made each load touch four times the cache lines).
__host__ __device__ constexpr int box_comps(int nf) { return nf + nf * (nf + 1) / 2; }
__host__ __device__ constexpr int box_pad(int nf) { return (box_comps(nf) + 3) / 4 * 4; }
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
    const float *ta = nullptr, *tb = nullptr;
    int cw = 0, ch = 0;
    Box a{}, b{};
};

// A table's sums over the box [x0, x1) × [y0, y1) clipped to the grid, all comps: four corner reads of
// whole entries, of which those on the grid's first row or column are zero and not made. Lanes of
// consecutive shifts read consecutive entries at the corners that move with the shift and one entry
// at those the grid's edge holds.
template <int NF>
__device__ __forceinline__ void box_read(float (&v)[box_pad(NF)], const float* __restrict__ t, int cw, int ch, int x0,
                                         int x1, int y0, int y1) {
    constexpr int NP = box_pad(NF);
    x0 = max(x0, 0), y0 = max(y0, 0), x1 = min(x1, cw), y1 = min(y1, ch);
#pragma unroll
    for (int i = 0; i < NP; ++i) v[i] = 0.f;
    if (x1 <= x0 || y1 <= y0) return;
    auto add = [&](int x, int y, float sign) {
        const float4* p = reinterpret_cast<const float4*>(t) + (size_t)(y - 1) * (NP / 4) * cw + (x - 1);
#pragma unroll
        for (int q = 0; q < NP / 4; ++q) {
            const float4 e = __ldg(p + (size_t)q * cw);
            v[4 * q] = fmaf(sign, e.x, v[4 * q]);
            v[4 * q + 1] = fmaf(sign, e.y, v[4 * q + 1]);
            v[4 * q + 2] = fmaf(sign, e.z, v[4 * q + 2]);
            v[4 * q + 3] = fmaf(sign, e.w, v[4 * q + 3]);
        }
    };
    // neighbouring corners first: each row's difference, then the difference of the rows
    if (x0 > 0 && y0 > 0) add(x0, y0, 1.f);
    if (y0 > 0) add(x1, y0, -1.f);
    if (x0 > 0) add(x0, y1, -1.f);
    add(x1, y1, 1.f);
}

}  // namespace zc
