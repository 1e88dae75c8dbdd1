// Moment sums of one side over the other side's image box, from summed-area tables.
//
// A map's correlations against the other side's weight plane w — a side's four feature sums and ten
// products, 14 of the 45 — are Σ plane(x + t)·w(x). Where w is 1 on a rectangle of grid cells and 0
// outside (the fixed image pasted whole; the moving one under a translation), that sum is the
// plane's sum over the rectangle moved by t: four reads of a summed-area table per shift instead of
// a plane's forward transforms, a product spectrum and two inverse passes. A 1024² pair at a
// translation transforms 18 correlations and 5 planes per side instead of 45 and 15: inverse columns
// 369 → 158 µs, inverse rows 393 → 169, forward rows 183 → 90, forward columns 240 → 85, for three
// launches of 21 + 33 + 44 µs a side beside them (each alone on the card). At a turned pose 32
// correlations and 5 + 15 planes are left.
//
// Precision: products f_i² are tabled less the weight (their mean over the image is 1 by the
// whitening; n is added back from the overlap), so entries stay near the field's own excursions. Sums
// within a tile are float32; those of the tiles and bands, the entries and a box's four corners are
// float64, so a sum's error scales with its own box, where a float32 transform's scales with both planes'
// energy: rms 0.04 (300² over 1000 × 900) to 0.8 (8² over 40²) of a transform's over 14 planes, blobs,
// ramps and flat halves. The score divides the sums by the exact number of pixels they cover. On 1800
// translations of pairs of 8 to 420 pixels a side, half of them ramps, steps or flat halves, the rms error of
// a map's cells is 0.61 of that with all 45 correlations transformed, and the argmax leaves the float64
// oracle's 17 times against 26; turned, 0.91 and 62 against 75. Float32 entries, and the transform's n, were not
// enough: 25 against 10 in 600 translations. They cost less, by 0.08 ms of a map of 1024² (score 262 against
// 313 µs, tables 78 against 98).
//
// Built from tiles of 32 columns × 8 rows, a warp each, in three launches, so that the table (112
// bytes a cell) is written once and the samples (20 bytes) are read twice: k_box_sums leaves each
// tile's column, row and total sums; k_box_scan turns them into what lies above, left and above-left
// of a tile; k_box_write walks a tile's rows with the columns' running sums in registers and scans
// each row across the lanes.
#include "box.cuh"
#include "common.cuh"
#include "kernels.hpp"

namespace zc {
namespace {

constexpr int kTile = 32;
constexpr int kRows = 8;   // short walks: tall tiles left the card waiting on a few warps' chains
constexpr int kWarps = 4;  // tiles per block, side by side

// a table's scratch: column sums [band][comp][x], row sums [y][tile][comp], totals [band][tile][comp]
struct BoxScratch {
    double *col, *row, *tot;
    int nband, ntile;
};
__host__ BoxScratch scratch(void* p, int nf, int cw, int ch) {
    const int nc = box_comps(nf);
    BoxScratch s;
    s.nband = (ch + kRows - 1) / kRows, s.ntile = (cw + kTile - 1) / kTile;
    s.col = static_cast<double*>(p);
    s.row = s.col + (size_t)s.nband * cw * nc;
    s.tot = s.row + (size_t)ch * s.ntile * nc;
    return s;
}

// the comps of one cell from its samples (w, w f_0 .. )
template <int NF>
__device__ __forceinline__ void comps_of(float (&v)[box_comps(NF)], const float (&s)[1 + NF]) {
    const float inv = s[0] > 1e-6f ? 1.f / s[0] : 0.f;
    float f[NF];
#pragma unroll
    for (int i = 0; i < NF; ++i) {
        v[i] = s[1 + i];
        f[i] = s[1 + i] * inv;
    }
#pragma unroll
    for (int k = 0; k < box_comps(NF) - NF; ++k) {
        const int i = box_i(k, NF), j = box_j(k, NF);
        v[NF + k] = s[1 + i] * f[j] - (i == j ? s[0] : 0.f);
    }
}

template <int NF>
__device__ __forceinline__ void load_cell(float (&s)[1 + NF], const float* __restrict__ grid, size_t gn, int cw, int x,
                                          int y, bool in) {
#pragma unroll
    for (int p = 0; p <= NF; ++p) s[p] = in ? __ldg(&grid[p * gn + (size_t)y * cw + x]) : 0.f;
}

// the warp's sums of 16 values: lane l returns the sum of value l / 2 (16 shuffles, not 80: each
// step adds and halves the values a lane still carries)
__device__ __forceinline__ float warp_sums16(const float (&v)[16]) {
    const int lane = threadIdx.x & 31;
    float a[8], b[4], c[2];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = ((lane & 16) ? v[8 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, (lane & 16) ? v[i] : v[8 + i], 16);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = ((lane & 8) ? a[4 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, (lane & 8) ? a[i] : a[4 + i], 8);
#pragma unroll
    for (int i = 0; i < 2; ++i) c[i] = ((lane & 4) ? b[2 + i] : b[i]) + __shfl_xor_sync(0xffffffffu, (lane & 4) ? b[i] : b[2 + i], 4);
    const float d = ((lane & 2) ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, (lane & 2) ? c[0] : c[1], 2);
    return d + __shfl_xor_sync(0xffffffffu, d, 1);
}

template <int NF>
__global__ void __launch_bounds__(32 * kWarps) k_box_sums(const float* __restrict__ grid, int cw, int ch, BoxScratch sc) {
    constexpr int NC = box_comps(NF);
    const int lane = threadIdx.x & 31, tile = blockIdx.x * kWarps + (threadIdx.x >> 5), b = blockIdx.y;
    if (tile >= sc.ntile) return;
    const int x = tile * kTile + lane;
    const size_t gn = (size_t)cw * ch;
    float s[kRows][1 + NF];
#pragma unroll
    for (int r = 0; r < kRows; ++r) load_cell<NF>(s[r], grid, gn, cw, x, b * kRows + r, x < cw && b * kRows + r < ch);
    float col[16], tot = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) col[c] = 0.f;
    const int comp = lane >> 1;
    const bool owner = (lane & 1) == 0 && comp < NC;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        float v[NC], w[16];
        comps_of<NF>(v, s[r]);
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            w[c] = c < NC ? v[c < NC ? c : 0] : 0.f;
            col[c] += w[c];
        }
        const float sum = warp_sums16(w);
        const int y = b * kRows + r;
        if (owner && y < ch) sc.row[((size_t)y * sc.ntile + tile) * NC + comp] = sum;
        tot += sum;
    }
    if (x < cw)
#pragma unroll
        for (int c = 0; c < NC; ++c) sc.col[((size_t)b * NC + c) * cw + x] = col[c];
    if (owner) sc.tot[((size_t)b * sc.ntile + tile) * NC + comp] = tot;
}

// exclusive scan of n values `step` apart by one thread, 16 loads in flight
__device__ __forceinline__ void scan_serial(double* p, int n, size_t step) {
    double a = 0.0;
    for (int i0 = 0; i0 < n; i0 += 16) {
        double v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = i0 + i < n ? p[(i0 + i) * step] : 0.0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (i0 + i < n) p[(i0 + i) * step] = a;
            a += v[i];
        }
    }
}

// In place: column sums → over the bands above; row sums → over the tiles to the left; tile totals →
// over the tiles above and to the left (block 0: rows of tiles, then columns).
__global__ void __launch_bounds__(256) k_box_scan(BoxScratch sc, int nc, int cw, int ch, int ncol, int nrow) {
    const int i = (blockIdx.x - 1) * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0) {
        for (int k = threadIdx.x; k < sc.nband * nc; k += blockDim.x)
            scan_serial(sc.tot + (size_t)(k / nc) * sc.ntile * nc + k % nc, sc.ntile, nc);
        __syncthreads();
        for (int k = threadIdx.x; k < sc.ntile * nc; k += blockDim.x) scan_serial(sc.tot + k, sc.nband, (size_t)sc.ntile * nc);
    } else if (i < ncol) {
        scan_serial(sc.col + i, sc.nband, (size_t)cw * nc);
    } else if (i - ncol < nrow) {
        const int k = i - ncol;
        scan_serial(sc.row + (size_t)(k / nc) * sc.ntile * nc + k % nc, sc.ntile, nc);
    }
}

template <int NF>
__global__ void __launch_bounds__(32 * kWarps) k_box_write(const float* __restrict__ grid, int cw, int ch, BoxScratch sc,
                                                           double* __restrict__ t) {
    constexpr int NC = box_comps(NF), NP = box_pad(NF);
    const int lane = threadIdx.x & 31, tile = blockIdx.x * kWarps + (threadIdx.x >> 5), b = blockIdx.y;
    if (tile >= sc.ntile) return;
    const int x = tile * kTile + lane;
    const size_t gn = (size_t)cw * ch;
    const bool in = x < cw;
    double left = lane < NC ? sc.tot[((size_t)b * sc.ntile + tile) * NC + lane] : 0.0;  // lane c: comp c
    // what lies above the band in the tile's columns up to this one; within it, this column down to the row
    double above[NC];
    float run[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        double u = in ? sc.col[((size_t)b * NC + c) * cw + x] : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double w = __shfl_up_sync(0xffffffffu, u, o);
            if (lane >= o) u += w;
        }
        above[c] = u;
        run[c] = 0.f;
    }
#pragma unroll 2
    for (int r = 0; r < kRows; ++r) {
        const int y = b * kRows + r;
        if (y >= ch) break;
        float s[1 + NF], v[NC];
        load_cell<NF>(s, grid, gn, cw, x, y, in);
        comps_of<NF>(v, s);
        if (lane < NC) left += sc.row[((size_t)y * sc.ntile + tile) * NC + lane];
        double o2[NP];
#pragma unroll
        for (int c = 0; c < NP; ++c) {
            o2[c] = 0.0;
            if (c >= NC) continue;
            run[c] += v[c];
            float u = run[c];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float w = __shfl_up_sync(0xffffffffu, u, o);
                if (lane >= o) u += w;
            }
            o2[c] = __shfl_sync(0xffffffffu, left, c) + (above[c] + (double)u);
        }
        if (in) {
            double2* p = reinterpret_cast<double2*>(t) + (size_t)y * (NP / 2) * cw + x;
#pragma unroll
            for (int q = 0; q < NP / 2; ++q) p[(size_t)q * cw] = make_double2(o2[2 * q], o2[2 * q + 1]);
        }
    }
}

template <int NF>
cudaError_t build(const float* grid, int cw, int ch, double* t, void* tmp, cudaStream_t st) {
    constexpr int NC = box_comps(NF);
    const BoxScratch sc = scratch(tmp, NF, cw, ch);
    const dim3 g((sc.ntile + kWarps - 1) / kWarps, sc.nband);
    k_box_sums<NF><<<g, 32 * kWarps, 0, st>>>(grid, cw, ch, sc);
    const int ncol = cw * NC, nrow = ch * NC;
    k_box_scan<<<1 + (ncol + nrow + 255) / 256, 256, 0, st>>>(sc, NC, cw, ch, ncol, nrow);
    k_box_write<NF><<<g, 32 * kWarps, 0, st>>>(grid, cw, ch, sc, t);
    return cudaGetLastError();
}

}  // namespace

size_t box_table_bytes(int nf, int cw, int ch) { return (size_t)box_pad(nf) * ch * cw * sizeof(double); }
size_t box_scratch_bytes(int nf, int cw, int ch) {
    const size_t nb = (ch + kRows - 1) / kRows, nt = (cw + kTile - 1) / kTile;
    return (nb * cw + ch * nt + nb * nt) * box_comps(nf) * sizeof(double);
}

cudaError_t box_table(const float* grid, int cw, int ch, int nf, double* t, void* tmp, cudaStream_t st) {
    return nf == 3 ? build<3>(grid, cw, ch, t, tmp, st) : build<4>(grid, cw, ch, t, tmp, st);
}

}  // namespace zc
