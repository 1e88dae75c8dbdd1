// The per-shift score of a map from its correlations' real planes, and the argmax.
//
// Plane k of an item is ny rows of 2·WP floats (the rows pass writes them over the half spectra). A
// block scores 256 shifts at a time, one a thread, of the padded rows laid end to end; while it does,
// the next 256 shifts' sums are copied to shared memory (cp.async, 16 bytes a copy), so the float64
// centring and Cholesky wait on no load of a plane and spend no instructions on its address. With moment
// tables (modes 1 and 2) a shift's 16 or 32 corner reads are plain loads in front of them. A 1296 ×
// 1536 map of 45 correlations: rows 403 + score 109 µs, against 3643 µs with the row's sums held in
// shared memory; the sweep's 104 maps of 192²: 455 + 144 against 608 µs.
#include "box.cuh"
#include "combine.cuh"
#include "common.cuh"
#include "kernels.hpp"

namespace zc {
namespace {

constexpr int kScoreThreads = 256;
constexpr int kScorePer = 4;  // shifts per thread: one argmax atomic per 1024 shifts

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Shifts of rows y0 .. y0 + rows − 1 (nx of each row's `pitch` floats) of item blockIdx.y: R + b·qbs
// and n00p[b] read, map + b·mbs written; best and zero_out may be null.
template <int NF, bool EXACT, bool CALIB, int MODE>
__global__ void __launch_bounds__(kScoreThreads, 2) k_score(const float* __restrict__ R, size_t pstride, int pitch, int nx,
                                                            int ny, int y0, int rows, CombineParams cp, BoxSums bx,
                                                            const double* __restrict__ n00p, float* __restrict__ map,
                                                            unsigned long long* best, float* zero_out, size_t qbs,
                                                            size_t mbs) {
    constexpr int NS = corr_slots<NF, EXACT, MODE>();
    constexpr CorrSource from = corr_source<NF == 1 ? 4 : NF, MODE>();
    extern __shared__ __align__(16) float sums[];  // [2][NS][kScoreThreads]
    R += (size_t)blockIdx.y * qbs + (size_t)y0 * pitch;
    map += (size_t)blockIdx.y * mbs;
    if (CALIB) read_area(cp);
    const double n00 = lag0_units(cp, n00p[blockIdx.y]);
    const int nn = rows * pitch, f0 = blockIdx.x * kScorePer * kScoreThreads;
    auto fetch = [&](int q) {
        const int f = f0 + q * kScoreThreads;
        if (q < kScorePer && f < nn) {
            float* dst = sums + (q & 1) * NS * kScoreThreads;
            for (int i = threadIdx.x; i < NS * (kScoreThreads / 4); i += kScoreThreads) {
                const int k = i / (kScoreThreads / 4), o = 4 * (i % (kScoreThreads / 4));
                if (f + o < nn) copy16(dst + k * kScoreThreads + o, R + (size_t)k * pstride + f + o);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float bv = -3.4e38f;
    uint32_t bi = 0xffffffffu;
    fetch(0);
#pragma unroll 1
    for (int q = 0; q < kScorePer; ++q) {
        fetch(q + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int m = f0 + q * kScoreThreads + threadIdx.x, yr = m / pitch, x = m - yr * pitch, y = y0 + yr;
        if (m < nn && x < nx) {
            const float* r = sums + (q & 1) * NS * kScoreThreads + threadIdx.x;
            const CombineParams cpr = row_params(cp, y, ny);
            auto fft = [&](int c) { return r[from.at[c] * kScoreThreads]; };
            float sc;
            if constexpr (MODE == 0) {
                sc = combine_t<NF, EXACT, CALIB>(fft, cpr, n00);
            } else {
                double n = (double)fft(0) * cpr.inv_nn;
                sc = 0.f;
                if (overlap_alive<CALIB>(n, cpr, n00)) {
                    // the lag: A's cells b + t against B's box, B's cells a − t against A's
                    const int tx = x <= nx / 2 ? x : x - nx, ty = y <= ny / 2 ? y : y - ny;
                    // The moments are those of whole pixels, and the score divides by their exact number:
                    // the boxes' common cells, or the transform's sum rounded. (The transform's error in
                    // n, cancelled against exact moments, was most of what flat parts' covariances had.)
                    if (MODE == 2)
                        n = (double)max(min(bx.b.x1 + tx, bx.a.x1) - max(bx.b.x0 + tx, bx.a.x0), 0) *
                            (double)max(min(bx.b.y1 + ty, bx.a.y1) - max(bx.b.y0 + ty, bx.a.y0), 0);
                    else n = rint(n);
                    float va[box_pad(NF)], vb[box_pad(NF)];
                    box_read<NF>(va, bx.ta, bx.cw, bx.ch, bx.b.x0 + tx, bx.b.x1 + tx, bx.b.y0 + ty, bx.b.y1 + ty);
                    if (MODE == 2)
                        box_read<NF>(vb, bx.tb, bx.cw, bx.ch, bx.a.x0 - tx, bx.a.x1 - tx, bx.a.y0 - ty, bx.a.y1 - ty);
                    const double scale = cpr.inv_nn * (1.0 / fmax(n, 1e-8));
                    sc = combine_smi<NF, EXACT, CALIB>(
                        [&](int c, double rn) -> double {
                            if (from.src[c] == 0) return (double)fft(c) * scale;
                            const double v = (double)(from.src[c] == 1 ? va[from.at[c]] : vb[from.at[c]]) * rn;
                            return from.diag[c] ? v + 1.0 : v;
                        },
                        n, cpr);
                }
            }
            const uint32_t idx = (uint32_t)y * (uint32_t)nx + (uint32_t)x;
            map[idx] = sc;
            if (sc > bv || (sc == bv && idx < bi)) {
                bv = sc;
                bi = idx;
            }
            if (idx == 0 && zero_out) *zero_out = sc;
        }
        __syncthreads();  // the buffer is refilled by the next pass's fetch
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

template <int NF, bool EXACT, bool CALIB, int MODE>
cudaError_t launch(const float2* Q, const MapGeom& g, const CombineParams& cp, const BoxSums& bx, const double* n00,
                   float* map, unsigned long long* best, float* zero, cudaStream_t st, int batch, size_t q_stride,
                   size_t map_stride, int y0, int rows) {
    const int per = kScoreThreads * kScorePer, nn = rows * 2 * g.WP;
    const size_t sm = (size_t)2 * corr_slots<NF, EXACT, MODE>() * kScoreThreads * sizeof(float);
    auto k = k_score<NF, EXACT, CALIB, MODE>;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k<<<dim3((nn + per - 1) / per, batch), kScoreThreads, sm, st>>>(reinterpret_cast<const float*>(Q), (size_t)2 * g.ny * g.WP,
                                                                     2 * g.WP, g.nx, g.ny, y0, rows, cp, bx, n00, map, best,
                                                                     zero, 2 * q_stride, map_stride);
    return cudaGetLastError();
}

}  // namespace

cudaError_t map_scores(const float2* Q, const MapGeom& g, const CombineParams& cp, const double* n00, float* map,
                       unsigned long long* best, float* zero, cudaStream_t st, int batch, size_t q_stride,
                       size_t map_stride, int y0, int rows, const BoxSums& bx) {
    if (rows < 0) rows = g.ny - y0;
    if (y0 < 0 || rows <= 0 || y0 + rows > g.ny || (bx.mode && (!cp.exact || cp.nf < 3))) return cudaErrorInvalidValue;
    auto go = [&](auto f) { return f(Q, g, cp, bx, n00, map, best, zero, st, batch, q_stride, map_stride, y0, rows); };
    if (cp.nf == 1) return go(launch<1, false, false, 0>);
    if (!cp.exact) return cp.nf == 4 ? go(launch<4, false, false, 0>) : go(launch<3, false, false, 0>);
    if (cp.nf == 4) {
        if (bx.mode == 2) return cp.calib ? go(launch<4, true, true, 2>) : go(launch<4, true, false, 2>);
        if (bx.mode == 1) return cp.calib ? go(launch<4, true, true, 1>) : go(launch<4, true, false, 1>);
        return cp.calib ? go(launch<4, true, true, 0>) : go(launch<4, true, false, 0>);
    }
    if (bx.mode == 2) return cp.calib ? go(launch<3, true, true, 2>) : go(launch<3, true, false, 2>);
    if (bx.mode == 1) return cp.calib ? go(launch<3, true, true, 1>) : go(launch<3, true, false, 1>);
    return cp.calib ? go(launch<3, true, true, 0>) : go(launch<3, true, false, 0>);
}

}  // namespace zc
