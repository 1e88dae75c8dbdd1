// The rotation × scale sweep's own kernels (the reference's shaders/sweep.wgsl): the stacks
// interleaved per pixel, each candidate's window of canvas cells packed from k×k bilinear taps
// together with its zero-lag overlap, and the peaks of each candidate's map. The transforms and
// the per-shift score between them are the shift map's kernels (shiftmap.cu), batched over
// candidates.
#include "common.cuh"
#include "kernels.hpp"

namespace zc {
namespace {

// The stacks as the taps read them: pixels (w, w f0, w f1, w f2) as float4, then w f3 as floats, both
// in tiles of 4 × 2 pixels (a 128-byte line of the first, a 32-byte sector of the second). A tap's
// lanes follow a turned line through the image; in rows of pixels each lane of a steep one is in a
// line of its own, and the lines per load, not the bytes, bound the pass (L1 84 % busy, 37 % of the
// issue slots). 3240 poses of a 512² pair: 10.25 ms in rows with cells straddling passes, 8.6 in whole
// passes and paired products, 7.3 in tiles; gathering the four f3 of a tap in one load as well gave 2 %
// for 60 % more memory. Pixel (x, y) is at
// tile_x(x) + tile_y(y, row), row = 8 · tiles across; pixels past the image's edge are never read.
__host__ __device__ __forceinline__ constexpr unsigned tile_row(int w) { return ((unsigned)w + 3) / 4 * 8; }
__host__ __device__ __forceinline__ constexpr size_t tile_cells(int w, int h) { return (size_t)tile_row(w) * (((unsigned)h + 1) / 2); }
__device__ __forceinline__ unsigned tile_x(unsigned x) { return x + (x & ~3u); }
__device__ __forceinline__ unsigned tile_y(unsigned y, unsigned row) { return 4 * y + (y >> 1) * (row - 8); }

__global__ void k_interleave(const float* __restrict__ stack, int w, int h, float4* __restrict__ il) {
    const int n = w * h;
    float* p4 = reinterpret_cast<float*>(il + tile_cells(w, h));
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int y = i / w;
        const unsigned o = tile_x(i - y * w) + tile_y(y, tile_row(w));
        il[o] = make_float4(stack[i], stack[(size_t)n + i], stack[2 * (size_t)n + i], stack[3 * (size_t)n + i]);
        p4[o] = stack[4 * (size_t)n + i];
    }
}

constexpr int kPackTaps = 6;  // the most taps per side that a sweep's cells take
// cells of a strip of k taps per side: whole passes of ⌊32/k⌋ cells
__host__ __device__ constexpr int pack_strip(int k) { return 32 / (32 / k) * (32 / k); }

// The K×K taps of a strip of W = pack_strip(K) cells (30 or 32) of a window's row, cells xw0 .. of canvas row cy;
// lane L < W returns cell xw0 + L's sums in s. The taps run across the lanes: in each pass, groups of
// K lanes take ⌊32/K⌋ cells, lane (g, tx) summing tap column tx of its cell over the K tap rows, so
// adjacent lanes read adjacent pixels (one cache line serves several lanes) instead of pixels a cell
// apart; the lane that owns a cell then adds its group's K column sums.
template <int K>
__device__ __forceinline__ void pack_cells(float (&s)[5], const float4* __restrict__ il, int sw, int sh, const float* P,
                                           const SweepCanvas& cv, int xw0, int win_x, int cy, int lane) {
    constexpr int CPW = 32 / K;
    const ulonglong2* u = reinterpret_cast<const ulonglong2*>(il);
    const float* p4 = reinterpret_cast<const float*>(il + tile_cells(sw, sh));  // the fifth plane
    const unsigned row = tile_row(sw);
    const float h0 = P[0], h1 = P[1], h2 = P[2], h3 = P[3], h4 = P[4], h5 = P[5], h6 = P[6], h7 = P[7], h8 = P[8];
    const bool affine = h6 == 0.f && h7 == 0.f && h8 == 1.f;  // qz is 1 then
    const float inv = 1.f / (float)(K * K);
    const int grp = lane / K, tx = lane - grp * K, cx0 = (int)P[10] + xw0;
    const unsigned wlim = (unsigned)(sw - 1), hlim = (unsigned)(sh - 1);
#pragma unroll 1
    for (int c0 = 0; c0 < pack_strip(K) && xw0 + c0 < win_x; c0 += CPW) {
        const int xw = xw0 + c0 + grp, cx = cx0 + c0 + grp;
        f32x2 a01 = 0, a23 = 0;
        float a4 = 0.f;
        if (grp < CPW && xw < win_x && cx < cv.G && cy < cv.G) {
            const float px = cv.ox + ((float)cx + ((float)tx + 0.5f) / (float)K) * cv.cell;
#pragma unroll
            for (int ty = 0; ty < K; ++ty) {
                const float py = cv.oy + ((float)cy + ((float)ty + 0.5f) / (float)K) * cv.cell;
                float qx = h0 * px + h1 * py + h2;
                float qy = h3 * px + h4 * py + h5;
                if (!affine) {
                    const float qz = h6 * px + h7 * py + h8;
                    if (fabsf(qz) < 1e-8f) continue;
                    if (qz != 1.f) qx = qx / qz, qy = qy / qz;
                }
                const float fx = qx - 1.0f, fy = qy - 1.0f;
                float flx, fly;
                const unsigned ix = floor_index(fx, flx), iy = floor_index(fy, fly);
                if (ix >= wlim || iy >= hlim) continue;  // x0 ≥ 0 and x0 + 1 < w
                const float ax = fx - flx, ay = fy - fly;
                const float w00 = (1.f - ax) * (1.f - ay), w10 = ax * (1.f - ay), w01 = (1.f - ax) * ay, w11 = ax * ay;
                const unsigned X0 = tile_x(ix), X1 = tile_x(ix + 1), Y0 = tile_y(iy, row), Y1 = tile_y(iy + 1, row);
                const unsigned i00 = X0 + Y0, i10 = X1 + Y0, i01 = X0 + Y1, i11 = X1 + Y1;
                const ulonglong2 p00 = __ldg(u + i00), p10 = __ldg(u + i10), p01 = __ldg(u + i01), p11 = __ldg(u + i11);
                const f32x2 v00 = pack2(w00, w00), v10 = pack2(w10, w10), v01 = pack2(w01, w01), v11 = pack2(w11, w11);
                a01 = add2(a01, fma2(v11, p11.x, fma2(v01, p01.x, fma2(v00, p00.x, mul2(v10, p10.x)))));
                a23 = add2(a23, fma2(v11, p11.y, fma2(v01, p01.y, fma2(v00, p00.y, mul2(v10, p10.y)))));
                a4 += w00 * __ldg(&p4[i00]) + w10 * __ldg(&p4[i10]) + w01 * __ldg(&p4[i01]) + w11 * __ldg(&p4[i11]);
            }
        }
        float a[5];
        unpack2(a01, a[0], a[1]);
        unpack2(a23, a[2], a[3]);
        a[4] = a4;
        // lane L owns cell L of the strip: this pass holds it when c0 ≤ L < c0 + CPW, in group L − c0
        const bool here = lane >= c0 && lane < c0 + CPW;
        const int src = here ? (lane - c0) * K : 0;
#pragma unroll
        for (int p = 0; p < 5; ++p) {
            float t = 0.f;
#pragma unroll
            for (int j = 0; j < K; ++j) t += __shfl_sync(0xffffffffu, a[p], src + j);
            if (here) s[p] = t * inv;
        }
    }
}

// Warp w of a block takes a strip of the cells (30 or 32) of row y of item z's window; the item's
// pose is poses[(slot0 + z)·12 ..]: the dest → source map (row-major 3×3, 1-based pixels), taps per
// side (1 to 6), the window's first canvas cell. The cell's value is the mean of k×k bilinear taps of
// the source stack at the cell's sub-points (sweep.wgsl tap, pack_sweep); a tap whose 2×2
// footprint leaves the image adds nothing. Cells past the G×G canvas are zero. Output plane-major
// [5][win_y][win_x] per item. With fixed weights fw ([Fy][Fx], the fixed window at canvas cell
// (fx0, fy0)) the item's zero-lag overlap Σ w_moving · w_fixed over the cells both windows cover
// accumulates into n0[z] (sweep.wgsl zero_lag reads the same value off the correlation of the weight planes).
__global__ void __launch_bounds__(256, 4) k_sweep_pack(const float4* __restrict__ il, int sw, int sh,
                                                       const float* __restrict__ poses, int slot0, int win_x, int win_y,
                                                       SweepCanvas cv, const float* __restrict__ fw, int fx0, int fy0,
                                                       int Fx, int Fy, float* __restrict__ grid, double* __restrict__ n0) {
    const int lane = threadIdx.x & 31;
    const int y = blockIdx.y * 8 + (threadIdx.x >> 5), z = blockIdx.z;
    const float* P = poses + (size_t)(slot0 + z) * 12;
    const int cy = (int)P[11] + y, k = min(max((int)P[9], 1), kPackTaps);
    const int strip = pack_strip(k), x0 = blockIdx.x * strip, x = x0 + lane;
    const bool in_win = lane < strip && x < win_x && y < win_y;
    float s[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    if (y < win_y) {
        switch (k) {
            case 1: pack_cells<1>(s, il, sw, sh, P, cv, x0, win_x, cy, lane); break;
            case 2: pack_cells<2>(s, il, sw, sh, P, cv, x0, win_x, cy, lane); break;
            case 3: pack_cells<3>(s, il, sw, sh, P, cv, x0, win_x, cy, lane); break;
            case 4: pack_cells<4>(s, il, sw, sh, P, cv, x0, win_x, cy, lane); break;
            case 5: pack_cells<5>(s, il, sw, sh, P, cv, x0, win_x, cy, lane); break;
            default: pack_cells<6>(s, il, sw, sh, P, cv, x0, win_x, cy, lane); break;
        }
    }
    if (in_win) {
        const size_t wn = (size_t)win_x * win_y;
        float* g = grid + (size_t)z * 5 * wn + (size_t)y * win_x + x;
#pragma unroll
        for (int p = 0; p < 5; ++p) g[p * wn] = s[p];
    }
    if (!n0) return;
    double v = 0.0;
    if (in_win) {
        const int fx = (int)P[10] + x - fx0, fy = cy - fy0;
        if (fx >= 0 && fy >= 0 && fx < Fx && fy < Fy) v = (double)s[0] * (double)__ldg(&fw[(size_t)fy * Fx + fx]);
    }
    __shared__ double red[32];
    v = block_sum(v, red);
    if (threadIdx.x == 0 && v != 0.0) atomicAdd(&n0[z], v);
}

// One block per item (sweep.wgsl peaks_sweep): lane l < 256 keeps the best 3×3 local maximum
// (periodic, > 0, the first of equal ones) among the shifts t ≡ l (mod 256); the n_peak best lanes
// (equal scores: the lower lane first) are written to slot (slot0 + z) as (score, index), and
// (0, 0xffffffff) where fewer lanes found one. The block's 1024 threads scan each lane's shifts
// four ways (thread (l, q) the shifts l + 256·(q + 4j)) and merge the four bests per lane by the
// same rule (higher score, then lower shift), which is the lane's own best.
__global__ void __launch_bounds__(1024) k_sweep_peaks(const float* __restrict__ maps, int nx, int ny, size_t mstride,
                                                      int n_peak, int slot0, float* __restrict__ ps,
                                                      uint32_t* __restrict__ pi) {
    const float* m = maps + (size_t)blockIdx.x * mstride;
    const int nn = nx * ny;
    const int l = threadIdx.x & 255, q = threadIdx.x >> 8;
    float bv = 0.f;
    uint32_t bi = 0xffffffffu;
    for (int t = l + 256 * q; t < nn; t += 1024) {
        const float v = __ldg(&m[t]);
        if (v <= bv) continue;
        const int y = t / nx, x = t - y * nx;
        const int ym = (y + ny - 1) % ny, yp = (y + 1) % ny, xm = (x + nx - 1) % nx, xp = (x + 1) % nx;
        const bool ok = !(__ldg(&m[ym * nx + xm]) > v || __ldg(&m[ym * nx + x]) > v || __ldg(&m[ym * nx + xp]) > v ||
                          __ldg(&m[y * nx + xm]) > v || __ldg(&m[y * nx + xp]) > v || __ldg(&m[yp * nx + xm]) > v ||
                          __ldg(&m[yp * nx + x]) > v || __ldg(&m[yp * nx + xp]) > v);
        if (ok) {
            bv = v;
            bi = (uint32_t)t;
        }
    }
    __shared__ float sv[3][256];
    __shared__ uint32_t si[3][256];
    if (q > 0) {
        sv[q - 1][l] = bv;
        si[q - 1][l] = bi;
    }
    __syncthreads();
    if (q == 0)
        for (int r = 0; r < 3; ++r) {
            const float v = sv[r][l];
            const uint32_t i = si[r][l];
            if (v > bv || (v == bv && i < bi)) {
                bv = v;
                bi = i;
            }
        }
    // a positive float's bits order like the float: (score, inverted lane) as one key
    unsigned long long key = (q > 0 || bi == 0xffffffffu)
                                 ? 0ull
                                 : ((unsigned long long)__float_as_uint(bv) << 32) | (0xffffffffu - (uint32_t)l);
    __shared__ unsigned long long wmax[32];
    __shared__ unsigned long long top;
    for (int k = 0; k < n_peak; ++k) {
        unsigned long long w = key;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, w, o);
            w = other > w ? other : w;
        }
        if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = w;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long b = 0;
            for (int i = 0; i < 32; ++i) b = wmax[i] > b ? wmax[i] : b;
            top = b;
        }
        __syncthreads();
        const unsigned long long b = top;
        const size_t o = (size_t)(slot0 + blockIdx.x) * n_peak + k;
        if (b == 0ull) {
            if (threadIdx.x == 0) {
                ps[o] = 0.f;
                pi[o] = 0xffffffffu;
            }
        } else if (b == key) {
            ps[o] = bv;
            pi[o] = bi;
            key = 0ull;
        }
        __syncthreads();
    }
}

}  // namespace

size_t sweep_interleaved_bytes(int w, int h) { return tile_cells(w, h) * 20; }

cudaError_t sweep_interleave(const float* stack, int w, int h, float4* il, cudaStream_t st) {
    int blocks = (w * h + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    k_interleave<<<blocks, 256, 0, st>>>(stack, w, h, il);
    return cudaGetLastError();
}

cudaError_t sweep_pack(const float4* il, int sw, int sh, const float* poses, int slot0, int batch, int win_x,
                       int win_y, const SweepCanvas& cv, const float* fw, int fx0, int fy0, int Fx, int Fy, float* grid,
                       double* n0, cudaStream_t st) {
    if (n0) {
        const cudaError_t e = cudaMemsetAsync(n0, 0, (size_t)batch * sizeof(double), st);
        if (e != cudaSuccess) return e;
    }
    dim3 g((win_x + 29) / 30, (win_y + 7) / 8, batch);  // strips of 30 cells at least
    k_sweep_pack<<<g, 256, 0, st>>>(il, sw, sh, poses, slot0, win_x, win_y, cv, fw, fx0, fy0, Fx, Fy, grid, n0);
    return cudaGetLastError();
}

cudaError_t sweep_peaks(const float* maps, int nx, int ny, size_t map_stride, int batch, int n_peak, int slot0,
                        float* ps, uint32_t* pi, cudaStream_t st) {
    k_sweep_peaks<<<batch, 1024, 0, st>>>(maps, nx, ny, map_stride, n_peak, slot0, ps, pi);
    return cudaGetLastError();
}

}  // namespace zc
