// The per-shift score of a map from its correlations' real planes, and the argmax.
//
// Plane k of an item is ny rows of 2·WP floats (the rows pass writes them over the half spectra), so
// a shift's sums are n_corr coalesced loads. One thread scores one shift: the float64 centring and
// Cholesky run at the occupancy their registers allow, with nothing else of the block waiting on
// them, and a warp whose 32 shifts are all under the overlap floor reads one sum each. A 1296 × 1536
// map of 45 correlations: rows 403 + score 109 µs, against 3643 µs with the row's sums held in
// shared memory; the sweep's 104 maps of 192²: 455 + 144 against 608 µs.
#include "combine.cuh"
#include "common.cuh"
#include "kernels.hpp"

namespace zc {
namespace {

constexpr int kScoreThreads = 256;
constexpr int kScorePer = 4;  // shifts per thread: one argmax atomic per 1024 shifts

// Shifts of rows y0 .. y0 + rows − 1 (nx per row) of item blockIdx.y: R + b·qbs and n00p[b] read,
// map + b·mbs written; best and zero_out may be null.
template <int NF, bool EXACT, bool CALIB>
__global__ void __launch_bounds__(kScoreThreads) k_score(const float* __restrict__ R, size_t pstride, int pitch, int nx,
                                                         int ny, int y0, int rows, CombineParams cp,
                                                         const double* __restrict__ n00p, float* __restrict__ map,
                                                         unsigned long long* best, float* zero_out, size_t qbs,
                                                         size_t mbs) {
    R += (size_t)blockIdx.y * qbs;
    map += (size_t)blockIdx.y * mbs;
    const double n00 = lag0_units(cp, n00p[blockIdx.y]);
    const int nn = rows * nx;
    float bv = -3.4e38f;
    uint32_t bi = 0xffffffffu;
#pragma unroll 1
    for (int q = 0; q < kScorePer; ++q) {
        const int m = (blockIdx.x * kScorePer + q) * kScoreThreads + threadIdx.x;
        if (m >= nn) break;
        const int y = y0 + m / nx, x = m - (y - y0) * nx;
        const float* r = R + (size_t)y * pitch + x;
        const float sc =
            combine_t<NF, EXACT, CALIB>([&](int k) { return __ldg(&r[(size_t)k * pstride]); }, row_params(cp, y, ny), n00);
        const uint32_t idx = (uint32_t)y * (uint32_t)nx + (uint32_t)x;
        map[idx] = sc;
        if (sc > bv || (sc == bv && idx < bi)) {
            bv = sc;
            bi = idx;
        }
        if (idx == 0 && zero_out) *zero_out = sc;
    }
    if (!best) return;
    unsigned long long key = (bi == 0xffffffffu) ? 0ull : argmax_key(bv, bi);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
        key = other > key ? other : key;
    }
    __shared__ unsigned long long wk[kScoreThreads / 32];
    if ((threadIdx.x & 31) == 0) wk[threadIdx.x >> 5] = key;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < kScoreThreads / 32; ++i) key = wk[i] > key ? wk[i] : key;
        if (key) atomicMax(best, key);
    }
}

template <int NF, bool EXACT, bool CALIB>
cudaError_t launch(const float2* Q, const MapGeom& g, const CombineParams& cp, const double* n00, float* map,
                   unsigned long long* best, float* zero, cudaStream_t st, int batch, size_t q_stride, size_t map_stride,
                   int y0, int rows) {
    const int per = kScoreThreads * kScorePer, nn = rows * g.nx;
    k_score<NF, EXACT, CALIB><<<dim3((nn + per - 1) / per, batch), kScoreThreads, 0, st>>>(
        reinterpret_cast<const float*>(Q), (size_t)2 * g.ny * g.WP, 2 * g.WP, g.nx, g.ny, y0, rows, cp, n00, map, best,
        zero, 2 * q_stride, map_stride);
    return cudaGetLastError();
}

}  // namespace

cudaError_t map_scores(const float2* Q, const MapGeom& g, const CombineParams& cp, const double* n00, float* map,
                       unsigned long long* best, float* zero, cudaStream_t st, int batch, size_t q_stride,
                       size_t map_stride, int y0, int rows) {
    if (rows < 0) rows = g.ny - y0;
    if (y0 < 0 || rows <= 0 || y0 + rows > g.ny) return cudaErrorInvalidValue;
    auto go = [&](auto f) { return f(Q, g, cp, n00, map, best, zero, st, batch, q_stride, map_stride, y0, rows); };
    if (cp.nf == 1) return go(launch<1, false, false>);
    if (cp.nf == 4) {
        if (!cp.exact) return go(launch<4, false, false>);
        return cp.calib ? go(launch<4, true, true>) : go(launch<4, true, false>);
    }
    if (!cp.exact) return go(launch<3, false, false>);
    return cp.calib ? go(launch<3, true, true>) : go(launch<3, true, false>);
}

}  // namespace zc
