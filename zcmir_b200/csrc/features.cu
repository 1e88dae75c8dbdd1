// Per-image SMI features (the reference's Smi.prepare, src/smi.zig:348-400):
// mean and spread → z → 256-bin histogram mid-rank → [r, r², Sobel |∇r|, fourth] → global ridge
// whitening → autocorrelation at |τ| ≤ 8 → the premultiplied stack [1, f0..f3].
//
// Per-pixel arithmetic is float32 with every operation rounded on its own in the reference's
// order (__fadd_rn & co. keep the compiler from fusing them), so the histogram bins and ranks
// match a float32 restatement bit for bit; the image-wide sums are float64 (the reference sums
// in float32).
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.hpp"

namespace zc {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float mean_of(const double* stats, int n) {
    return __double2float_rn(stats[0] / (double)n);
}
__device__ __forceinline__ float spread_of(const double* stats, int n) {
    return __double2float_rn(sqrt(fmax(stats[1] / (double)n, 1e-12)));
}

// f16 texels and back (src/gls.zig:433-442 with half precision)
__global__ void k_quant_half(float* g, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        g[i] = __half2float(__float2half_rn(g[i]));
}

// Σg (shaders/smi.wgsl:520-529 reduce1, float64 here)
__global__ void k_sum(const float* __restrict__ g, int n, double* stats) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc += (double)g[i];
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) atomicAdd(&stats[0], acc);
}

// Σ(g − mean)² with g − mean rounded to f32 (zscore_p then feat_moments, smi.wgsl:1548-1570)
__global__ void k_sumsq(const float* __restrict__ g, int n, double* stats) {
    __shared__ double sh[32];
    const float mean = mean_of(stats, n);
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double d = (double)__fsub_rn(g[i], mean);
        acc += d * d;
    }
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) atomicAdd(&stats[1], acc);
}

__device__ __forceinline__ unsigned bin_of(float g, float mean, float spread) {
    const float z = __fdiv_rn(__fsub_rn(g, mean), fmaxf(spread, 1e-8f));
    const float x = __fmul_rn(__fadd_rn(z, 4.0f), 32.0f);
    return (unsigned)fminf(fmaxf(x, 0.0f), 255.0f);
}

// 256-bin histogram of z over [−4, 4] (smi.wgsl:393-399)
__global__ void k_hist(const float* __restrict__ g, int n, const double* stats, unsigned* hist) {
    __shared__ unsigned sh[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    const float mean = mean_of(stats, n), spread = spread_of(stats, n);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&sh[bin_of(g[i], mean, spread)], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// mid-rank r = (cdf[b] + ½hist[b]) / N · 2 − 1 (smi.wgsl:401-420); every block scans the
// 256 bins itself, a thread a bin (one thread's walk over them was most of the launch)
__global__ void __launch_bounds__(kThreads) k_rank(const float* __restrict__ g, int n, const double* stats,
                                                const unsigned* __restrict__ hist, float* __restrict__ rank) {
    static_assert(kThreads == 256, "a thread per bin");
    __shared__ unsigned sh_h[256], sh_c[256], sh_w[8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned own = hist[threadIdx.x];
    unsigned c = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, c, o);
        if (lane >= o) c += v;
    }
    if (lane == 31) sh_w[wid] = c;
    __syncthreads();
    unsigned all = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (i < wid) c += sh_w[i];
        all += sh_w[i];
    }
    sh_h[threadIdx.x] = own;
    sh_c[threadIdx.x] = c - own;
    __syncthreads();
    const unsigned sh_tot = all > 0 ? all : 1u;
    const float mean = mean_of(stats, n), spread = spread_of(stats, n);
    const float tot = (float)sh_tot;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned b = bin_of(g[i], mean, spread);
        const float c = __fadd_rn((float)sh_c[b], __fmul_rn(0.5f, (float)sh_h[b]));
        rank[i] = __fsub_rn(__fmul_rn(__fdiv_rn(c, tot), 2.0f), 1.0f);
    }
}

// global ridge whitening L⁻¹ and μ (smi.wgsl:553-585), float64, stored as f32; mom: Σx_i (4), then
// Σx_i x_j for j ≤ i, row by row (10)
__device__ void whitening(const double (&mom)[14], int n, float ridge, float* wt) {
    const double nn = fmax((double)n, 1.0);
    double mu[4], G[16], L[16], X[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) mu[i] = mom[i] / nn;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) G[i * 4 + j] = mom[4 + i * (i + 1) / 2 + j] / nn - mu[i] * mu[j];
    double tr = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) tr += G[i * 5];
    const double rg = (double)ridge * fmax(tr * 0.25, 1e-12);
#pragma unroll
    for (int i = 0; i < 4; ++i) G[i * 5] += rg;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double s = G[i * 4 + j];
#pragma unroll
            for (int k = 0; k < j; ++k) s -= L[i * 4 + k] * L[j * 4 + k];
            if (i == j) L[i * 5] = sqrt(fmax(s, 1e-12));
            else L[i * 4 + j] = s / L[j * 5];
        }
#pragma unroll
    for (int col = 0; col < 4; ++col)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            double s = (i == col) ? 1.0 : 0.0;
#pragma unroll
            for (int k = 0; k < i; ++k) s -= L[i * 4 + k] * X[k * 4 + col];
            X[i * 4 + col] = s / L[i * 5];
        }
#pragma unroll
    for (int i = 0; i < 16; ++i) wt[i] = (float)X[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) wt[16 + i] = (float)mu[i];
}

// [r, r², Sobel |∇r|, fourth] with clamp-to-edge borders (smi.wgsl:422-462), and with them Σx_i (4)
// and the lower triangle of Σx_i x_j (10) in float64 (smi.wgsl:531-551), which the last block turns
// into the whitening. Small images are latency: the features, their moments and the one-thread
// Cholesky as three launches took 16 µs of a 256² side's build (now 8), the last two mostly 40 barriers and
// a chain through local memory. stats: [2..15] the moments, [16] the blocks done (all zeroed before).
constexpr int kFeatRows = 8, kFeatMoms = 14;
__global__ void __launch_bounds__(32 * kFeatRows) k_feats(const float* __restrict__ r, int w, int h, int mode,
                                                          float* __restrict__ feat, float* __restrict__ mag, double* stats,
                                                          float* __restrict__ wt) {
    const size_t n = (size_t)w * h;
    const int tx = (w + 31) / 32, tiles = tx * ((h + kFeatRows - 1) / kFeatRows);
    double a[kFeatMoms];
#pragma unroll
    for (int k = 0; k < kFeatMoms; ++k) a[k] = 0.0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int x = tile % tx * 32 + (threadIdx.x & 31), y = tile / tx * kFeatRows + (threadIdx.x >> 5);
        if (x >= w || y >= h) continue;
        auto t = [&](int dx, int dy) {
            const int xx = min(max(x + dx, 0), w - 1), yy = min(max(y + dy, 0), h - 1);
            return __ldg(&r[(size_t)yy * w + xx]);
        };
        const float c = t(0, 0);
        float gx = __fadd_rn(-t(-1, -1), t(1, -1));
        gx = __fsub_rn(gx, __fmul_rn(2.0f, t(-1, 0)));
        gx = __fadd_rn(gx, __fmul_rn(2.0f, t(1, 0)));
        gx = __fsub_rn(gx, t(-1, 1));
        gx = __fadd_rn(gx, t(1, 1));
        float gy = __fsub_rn(-t(-1, -1), __fmul_rn(2.0f, t(0, -1)));
        gy = __fsub_rn(gy, t(1, -1));
        gy = __fadd_rn(gy, t(-1, 1));
        gy = __fadd_rn(gy, __fmul_rn(2.0f, t(0, 1)));
        gy = __fadd_rn(gy, t(1, 1));
        const float g = __fsqrt_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)));
        float f3 = 0.0f;
        if (mode == 0) {
            f3 = __fadd_rn(__fadd_rn(__fadd_rn(t(-1, 0), t(1, 0)), t(0, -1)), t(0, 1));
            f3 = __fsub_rn(f3, __fmul_rn(4.0f, c));
        } else if (mode == 2) {
            f3 = __fmul_rn(__fmul_rn(c, c), c);
        }
        const size_t i = (size_t)y * w + x;
        const float f[4] = {c, __fmul_rn(c, c), g, f3};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            feat[(size_t)p * n + i] = f[p];
            a[p] += (double)f[p];
#pragma unroll
            for (int q = 0; q <= p; ++q) a[4 + p * (p + 1) / 2 + q] += (double)f[p] * (double)f[q];
        }
        mag[i] = g;
    }
    __shared__ double part[kFeatRows][kFeatMoms];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kFeatMoms; ++k) {
        const double v = warp_sum(a[k]);
        if (lane == 0) part[wid][k] = v;
    }
    __syncthreads();
    if (wid != 0) return;
    if (lane < kFeatMoms) {
        double v = 0.0;
#pragma unroll
        for (int i = 0; i < kFeatRows; ++i) v += part[i][lane];
        atomicAdd(&stats[2 + lane], v);
        __threadfence();
    }
    __syncwarp();
    if (lane != 0) return;
    unsigned* done = reinterpret_cast<unsigned*>(&stats[2 + kFeatMoms]);
    if (atomicAdd(done, 1u) != gridDim.x - 1) return;
    __threadfence();
    double mom[kFeatMoms];
#pragma unroll
    for (int k = 0; k < kFeatMoms; ++k) mom[k] = __ldcg(&stats[2 + k]);
    whitening(mom, (int)n, 1e-4f, wt);
}

// x ← L⁻¹(x − μ), products rounded one by one in j order (smi.wgsl:587-599), in all the places the
// features are kept: by plane, by pixel (feat4), and the stack [w, w f0..w f3] with w = 1
// (smi.wgsl:608-624)
__global__ void k_whiten(float* __restrict__ feat, int n, const float* __restrict__ wt, float4* __restrict__ feat4,
                         float* __restrict__ stack) {
    __shared__ float X[20];
    if (threadIdx.x < 20) X[threadIdx.x] = wt[threadIdx.x];
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float d[4], f[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) d[p] = __fsub_rn(feat[(size_t)p * n + i], X[16 + p]);
        stack[i] = 1.0f;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            f[p] = __fmul_rn(X[p * 4], d[0]);
#pragma unroll
            for (int q = 1; q < 4; ++q) f[p] = __fadd_rn(f[p], __fmul_rn(X[p * 4 + q], d[q]));
            feat[(size_t)p * n + i] = f[p];
            stack[(size_t)(p + 1) * n + i] = f[p];
        }
        feat4[i] = make_float4(f[0], f[1], f[2], f[3]);
    }
}

// Autocorrelation partial sums (smi.wgsl:935-975): one block per 32×32 tile with an 8-px halo in
// shared memory (zero outside the image, so a pair with either pixel outside adds nothing and
// every lag sums exactly the pairs inside the image). A lag and its negative sum the same pairs, so
// only the 153 lags with dy ≥ 0 are formed (the negative ones mirrored at the end). Register-blocked:
// thread (plane p, row lag dy, row group g) takes the tile rows g, g + 8, …, and walks each in steps of
// 8 columns with their 8 values and the 24 of the partner row at dy that the 17 column lags pair them
// with in registers, 16 of which the next step keeps (544 FMAs per 20 vector shared loads). Rows are
// 52 floats apart: at 48 the 8 rows that a quarter of a warp reads lay in two groups of banks and the
// loads, not the FMAs, bound the kernel (1024 × 768: 43 → 30 µs, with the columns taken in steps). The row groups' f32 sums are added in shared
// memory; partials [tile][153][4].
constexpr int kAcfTile = 32, kAcfHalo = 8, kAcfSpan = kAcfTile + 2 * kAcfHalo, kAcfHigh = kAcfTile + kAcfHalo, kAcfGroups = 8;
constexpr int kAcfThreads = 4 * 9 * kAcfGroups;  // 288
constexpr int kAcfPitch = kAcfSpan + 4, kAcfPlane = kAcfHigh * kAcfPitch;

__global__ void __launch_bounds__(kAcfThreads) k_acf(const float* __restrict__ feat, int w, int h,
                                                     float* __restrict__ part) {
    __shared__ __align__(16) float sh[4 * kAcfPlane];
    const int x0 = blockIdx.x * kAcfTile, y0 = blockIdx.y * kAcfTile;
    const size_t n = (size_t)w * h;
    for (int k = threadIdx.x; k < kAcfHigh * kAcfSpan; k += blockDim.x) {
        const int x = k % kAcfSpan, y = k / kAcfSpan, gx = x0 - kAcfHalo + x, gy = y0 + y;
        const bool in = gx >= 0 && gx < w && gy < h;
        const size_t i = in ? (size_t)gy * w + gx : 0;
#pragma unroll
        for (int p = 0; p < 4; ++p) sh[p * kAcfPlane + y * kAcfPitch + x] = in ? feat[p * n + i] : 0.0f;
    }
    __syncthreads();
    const int g = threadIdx.x % kAcfGroups, dy = (threadIdx.x / kAcfGroups) % 9, p = threadIdx.x / (kAcfGroups * 9);
    const float* pl = sh + p * kAcfPlane;
    float acc[17];
#pragma unroll
    for (int d = 0; d < 17; ++d) acc[d] = 0.f;
    for (int ty = g; ty < kAcfTile; ty += kAcfGroups) {
        const float4* ar = reinterpret_cast<const float4*>(pl + ty * kAcfPitch + kAcfHalo);
        const float4* br = reinterpret_cast<const float4*>(pl + (ty + dy) * kAcfPitch);
        auto take = [](float* to, const float4& v) { to[0] = v.x, to[1] = v.y, to[2] = v.z, to[3] = v.w; };
        float a[8], b[24];  // columns x .. x + 7; partner columns x − 8 .. x + 15
#pragma unroll
        for (int q = 0; q < 4; ++q) take(b + 4 * q, br[q]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            take(a, ar[2 * c]), take(a + 4, ar[2 * c + 1]);
            take(b + 16, br[4 + 2 * c]), take(b + 20, br[5 + 2 * c]);
#pragma unroll
            for (int x = 0; x < 8; ++x)
#pragma unroll
                for (int d = 0; d < 17; ++d) acc[d] = fmaf(a[x], b[x + d], acc[d]);
#pragma unroll
            for (int x = 0; x < 16; ++x) b[x] = b[x + 8];
        }
    }
    __syncthreads();
    // the row groups' sums: red[g][p·153 + lag] in the (now free) staging array
    float* red = sh;
#pragma unroll
    for (int d = 0; d < 17; ++d) red[g * kAcfSums + p * 153 + dy * 17 + d] = acc[d];
    __syncthreads();
    const size_t o = (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * kAcfSums;
    for (int k = threadIdx.x; k < kAcfSums; k += blockDim.x) {
        const int lag = k >> 2, pp = k & 3;
        float s = 0.f;
#pragma unroll
        for (int gg = 0; gg < kAcfGroups; ++gg) s += red[gg * kAcfSums + pp * 153 + lag];
        part[o + k] = s;
    }
}

// Σ over tiles (float64), ÷ the lag's pair count → acf[289][4] (not yet normalised), the lag and its
// negative
__global__ void k_acf_finish(const float* __restrict__ part, int ntiles, int w, int h, double* acf) {
    __shared__ double sh[32];
    const int k = blockIdx.x;  // lag·4 + plane
    double acc = 0.0;
    for (int t = threadIdx.x; t < ntiles; t += blockDim.x) acc += (double)part[(size_t)t * kAcfSums + k];
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) {
        const int lag = k / 4, dx = lag % 17 - 8, dy = lag / 17;
        const double cnt = fmax((double)(w - abs(dx)) * (double)(h - dy), 1.0);
        const double v = (w > abs(dx) && h > dy) ? acc / cnt : 0.0;
        acf[((8 + dy) * 17 + 8 + dx) * 4 + (k & 3)] = v;
        if (dy > 0) acf[((8 - dy) * 17 + 8 - dx) * 4 + (k & 3)] = v;
    }
}

// the pair's Bartlett correlation area (smi.wgsl:1572-1595) from both images' sums
__global__ void __launch_bounds__(320) k_pair_area(const double* __restrict__ a, const double* __restrict__ b,
                                                   double per_cell, double* area) {
    __shared__ double sh[32];
    double s = 0.0;
    if (threadIdx.x < 289) {
        double ra = 0.0, rb = 0.0;
        for (int i = 0; i < 4; ++i) {
            ra += a[threadIdx.x * 4 + i] / fmax(a[144 * 4 + i], 1e-12);
            rb += b[threadIdx.x * 4 + i] / fmax(b[144 * 4 + i], 1e-12);
        }
        s = ra * rb;
    }
    s = block_sum(s, sh);
    if (threadIdx.x == 0) *area = fmax(1.0, fmax(1.0, s / 16.0) * per_cell);
}

// Blocks of a launch over n pixels: one a pixel per thread, up to 8 per SM; the sums', whose blocks end
// in atomic additions to the same few places, at most two per SM
int grid_for(int n) {
    const int b = (n + kThreads - 1) / kThreads;
    return b < 148 * 8 ? (b > 0 ? b : 1) : 148 * 8;
}

int sum_grid(int n) { return grid_for(n) < 148 * 2 ? grid_for(n) : 148 * 2; }

}  // namespace

cudaError_t build_features(float* gray, int w, int h, int mode, bool half, float* rank, float* feat, float4* feat4,
                           float* mag, float* stack, FeatScratch& s, cudaStream_t st) {
    const int n = w * h;
    const int gb = grid_for(n), gs = sum_grid(n), tiles = ((w + 31) / 32) * ((h + kFeatRows - 1) / kFeatRows);
    static_assert(2 + kFeatMoms < kFeatStats, "the moments and the count of blocks done");
    cudaMemsetAsync(s.stats, 0, kFeatStats * sizeof(double), st);
    cudaMemsetAsync(s.hist, 0, 256 * sizeof(unsigned), st);
    if (half) k_quant_half<<<gb, kThreads, 0, st>>>(gray, n);
    k_sum<<<gs, kThreads, 0, st>>>(gray, n, s.stats);
    k_sumsq<<<gs, kThreads, 0, st>>>(gray, n, s.stats);
    k_hist<<<gs, kThreads, 0, st>>>(gray, n, s.stats, s.hist);
    k_rank<<<gb, kThreads, 0, st>>>(gray, n, s.stats, s.hist, rank);
    k_feats<<<std::min(tiles, 148 * 4), 32 * kFeatRows, 0, st>>>(rank, w, h, mode, feat, mag, s.stats, s.wt);
    k_whiten<<<gb, kThreads, 0, st>>>(feat, n, s.wt, feat4, stack);
    return cudaGetLastError();
}

cudaError_t autocorrelation(const float* feat, int w, int h, FeatScratch& s, cudaStream_t st) {
    dim3 ga((w + kAcfTile - 1) / kAcfTile, (h + kAcfTile - 1) / kAcfTile);
    const int ntiles = ga.x * ga.y;
    if ((size_t)ntiles * kAcfSums > s.acf_part_cap) return cudaErrorInvalidValue;
    k_acf<<<ga, kAcfThreads, 0, st>>>(feat, w, h, s.acf_part);
    k_acf_finish<<<kAcfSums, kThreads, 0, st>>>(s.acf_part, ntiles, w, h, s.acf);
    return cudaGetLastError();
}

cudaError_t pair_area_cells(const double* acf_a, const double* acf_b, double gcell, double* area, cudaStream_t st) {
    k_pair_area<<<1, 320, 0, st>>>(acf_a, acf_b, 1.0 / (gcell * gcell), area);
    return cudaGetLastError();
}

}  // namespace zc
