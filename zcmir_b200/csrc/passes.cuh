// The four passes of a shift map (and of a batch of sweep candidates' maps) as kernels templated
// on the line-FFT policy, with one launcher per pass. Included by the translation units that
// instantiate them for their line lengths (shiftmap.cu, lines_*.cu); everything here has internal
// linkage, so each unit carries its own instantiations.
//
//   forward rows   real planes → row R2C (rows < ch) into the half spectra [n_real][ny][WP]
//   forward cols   column FFTs of the half spectra, in place (rows ≥ ch read as zero)
//   inverse cols   per correlation and column tile: A·conj(B), inverse column FFT → Q[slot]
//   rows           per row: correlations paired as c1 + i·c2 on the Hermitian full row, inverse
//                  row FFT, the two real rows written over the half spectra they came from
//
// The per-shift score reads those real rows in a pass of its own (score.cu): it needs every
// correlation of a shift at once, and holding a row of all of them on chip left one block per SM
// whose float64 score could not overlap its transforms.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "kernels.hpp"

namespace zc {

// Line pitch of a column tile. Lines of 1024 points and more come in tiles of at most 8 lines
// (512 threads of N/16) and keep line_pitch's ≡ 4 (mod 16), a compile-time constant for
// compile-time lines; shorter lines come in wider tiles (the sweep's 192-point columns: 16 lines)
// whose half-warps touch 16 lines at one point each, which tile_pitch's odd pitch spreads over all
// bank pairs (≡ 4 put them in 4).
__host__ __device__ __forceinline__ constexpr int col_pitch(int n, int tx) {
    return n >= 1024 ? line_pitch(n) : tile_pitch(n, tx);
}

enum class Pass { FwdRows, FwdCols, InvCols, Rows };

// Everything a pass launch needs; the batch's items sit at the given strides (elements).
struct PassArgs {
    MapGeom g{};
    const CorrPlanDev* plan = nullptr;
    int batch = 1;
    const float* grid = nullptr;  // forward rows: [5][ch][cw] per item
    size_t grid_stride = 0;
    float2* half = nullptr;       // forward rows / columns: written; inverse columns: A
    size_t half_stride = 0;
    const float2* half_b = nullptr;  // inverse columns: B (b_stride 0: one fixed side)
    size_t b_stride = 0;
    float2* Q = nullptr;          // inverse columns: written; rows: transformed in place
    size_t q_stride = 0;
    int S = 1;                    // rows: the split
    const float2* tw_nx = nullptr;
};

namespace {

// ── forward: real planes → row R2C → column FFT ─────────────────────────────────────────────

// Real correlation plane r of a staged row: rows 0..4 the premultiplied samples s = [w, w f0..w f3],
// rows 5..8 f_i = s_{1+i} / s_0 (0 where s_0 ≤ 1e-6) (smi.wgsl:641-649): planes 0 → w, 1..4 → w f_i,
// 5..14 → s_i f_j. p: its samples' row, q: the row it is multiplied by (null for planes 0..4). RECIP: row 5
// is 1 / s_0 in place of the f_i, multiplied in at each use (the same products, rounded the same).
template <bool RECIP>
struct RealPlane {
    const float *p, *q, *inv;
    __device__ __forceinline__ RealPlane(int r, const float* row, int cw) : p(row + r * cw), q(nullptr), inv(row + 5 * cw) {
        if (r < 5) return;
        const int k = r - 5;
        const int ti = (k < 4) ? 0 : (k < 7) ? 1 : (k < 9) ? 2 : 3;
        const int tj = (k < 4) ? k : (k < 7) ? k - 3 : (k < 9) ? k - 5 : 3;
        p = row + (1 + ti) * cw;
        q = row + ((RECIP ? 1 : 5) + tj) * cw;
    }
    __device__ __forceinline__ float operator()(int x) const {
        if (!q) return p[x];
        return RECIP ? __fmul_rn(p[x], __fmul_rn(q[x], inv[x])) : p[x] * q[x];
    }
};

// shared memory a block may ask for, less the row kernel's own static array
constexpr size_t kRowShared = 227 * 1024 - 64;

// One block per grid row y < ch; lines = packed plane pairs (2z, 2z+1), lpb of them at a time.
// The row's samples are staged in shared memory once (after the line buffers).
// Batched over blockIdx.y: item b reads grid + b·gbs and writes half + b·hbs.
// LO: cw ≤ nx/2, so the first butterflies read only the row's lower half. RECIP: as RealPlane.
template <class F, bool LO, bool RECIP>
__global__ void __launch_bounds__(512, 1) k_fwd_rows(const float* __restrict__ grid, int cw, int ch, int WP,
                                                     CorrPlanDev plan, F f, int lpb, int products,
                                                     float2* __restrict__ half, size_t pstride, size_t gbs,
                                                     size_t hbs) {
    extern __shared__ float2 smem[];
    const int nx = f.n(), tl = f.tl();
    const int y = blockIdx.x;
    grid += (size_t)blockIdx.y * gbs;
    half += (size_t)blockIdx.y * hbs;
    const int line = threadIdx.x / tl;
    const int t = threadIdx.x - line * tl;
    const int pl = padded_len(nx);
    float2* buf = smem + (line < lpb ? line : 0) * pl;
    float* row = reinterpret_cast<float*>(smem + lpb * pl);  // [9][cw], [6][cw] or [5][cw] (RealPlane)
    __shared__ int planes[16];
    if (threadIdx.x < 16) planes[threadIdx.x] = threadIdx.x < plan.n_real ? plan.planes[threadIdx.x] : -1;
    const size_t gn = (size_t)cw * ch;
    for (int x = threadIdx.x; x < cw; x += blockDim.x) {
        float v[5];
#pragma unroll
        for (int p = 0; p < 5; ++p) row[p * cw + x] = v[p] = __ldg(&grid[p * gn + (size_t)y * cw + x]);
        if (products) {
            const float inv = v[0] <= 1e-6f ? 0.f : 1.f / v[0];
            if (RECIP) row[5 * cw + x] = inv;
            else
#pragma unroll
                for (int p = 1; p < 5; ++p) row[(4 + p) * cw + x] = v[p] * inv;
        }
    }
    __syncthreads();
    const int n_cplx = (plan.n_real + 1) / 2;
    for (int z0 = 0; z0 < n_cplx; z0 += lpb) {
        const int z = z0 + line;
        const bool act = line < lpb && z < n_cplx;
        const bool has_b = act && 2 * z + 1 < plan.n_real;
        const RealPlane<RECIP> ra(act ? planes[2 * z] : 0, row, cw), rb(has_b ? planes[2 * z + 1] : 0, row, cw);
        // the first butterflies read the staged rows directly (real planes ra + i·rb, zero past cw)
        f.fresh().template run_in<false, LO>(buf, t, act, [&](int x) {
            float2 v = make_float2(0.f, 0.f);
            if (x < cw) {
                v.x = ra(x);
                if (has_b) v.y = rb(x);
            }
            return v;
        });
        if (act) {
            float2* oa = half + (size_t)(2 * z) * pstride + (size_t)y * WP;
            float2* ob = half + (size_t)(2 * z + 1) * pstride + (size_t)y * WP;
            for (int x = t; x <= nx / 2; x += tl) {
                const float2 Z = buf[pad_idx(x)];
                const float2 Zm = buf[pad_idx(x == 0 ? 0 : nx - x)];
                oa[x] = make_float2(0.5f * (Z.x + Zm.x), 0.5f * (Z.y - Zm.y));
                if (has_b) ob[x] = make_float2(0.5f * (Z.y + Zm.y), 0.5f * (Zm.x - Z.x));
            }
        }
        __syncthreads();
    }
}

// Column FFTs of the half spectra, in place: block = a tile of tx columns of one plane; rows
// ≥ rows_in read as zero. Thread (column c, line thread t), c fastest, so each load or store of
// a warp covers 8 rows × 4 adjacent columns (whole 32-byte sectors); the first butterflies read
// global memory and the last write it (run_io), with only the middle stages in shared memory. With
// npad the planes' columns lie end to end, npad to a plane, and tiles cross from one to the next.
// LO: rows_in ≤ n/2, so the first butterflies read only rows y < n/2 (the rest are zero).
template <class F, bool INV, bool LO, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_cols(float2* __restrict__ half, size_t pstride, int WP, int ncols,
                                                 int npad, int planes, int rows_in, F f, int txr) {
    extern __shared__ float2 smem[];
    const int tx = F::kTx && MINB > 1 ? F::kTx : txr;  // (a constant cost 3072 points 8 %)
    const int pl = col_pitch(f.n(), tx);
    const int c = threadIdx.x % tx, t = threadIdx.x / tx;
    int plane = blockIdx.y, col = blockIdx.x * tx + c;
    if (npad) {
        plane = col / npad;
        col -= plane * npad;
    }
    const bool okc = plane < planes && col < ncols;
    float2* p = half + (size_t)(okc ? plane : 0) * pstride + col;
    f.template run_io<INV, LO>(
        smem + c * pl, t, true,
        [&](int y) { return (okc && y < rows_in) ? p[(size_t)y * WP] : make_float2(0.f, 0.f); },
        [&](int y, float2 v) {
            if (okc) p[(size_t)y * WP] = v;
        });
}

// ── inverse: products and column IFFTs ──────────────────────────────────────────────────────

// block (correlation slot k, column tile, item): P = A·conj(B) on the tile, inverse column FFT
// → Q; item b reads ha + b·abs, hb + b·bbs and writes Q + b·qbs. npad: as k_cols, over the correlations.
template <class F, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_inv_cols(const float2* __restrict__ ha, const float2* __restrict__ hb,
                                                     size_t pstride, int WP, int ncols, int npad, CorrPlanDev plan, F f, int txr,
                                                     float2* __restrict__ Q, size_t abs_, size_t bbs, size_t qbs) {
    extern __shared__ float2 smem[];
    const size_t item = blockIdx.z;
    const int tx = F::kTx ? F::kTx : txr;
    const int c = threadIdx.x % tx, t = threadIdx.x / tx;
    int k = blockIdx.x, col = blockIdx.y * tx + c;
    if (npad) {
        k = (blockIdx.x * tx + c) / npad;
        col = blockIdx.x * tx + c - k * npad;
    }
    const bool okc = k < plan.n_corr && col < ncols;
    if (!okc) k = 0;
    const float2* A = ha + item * abs_ + (size_t)plan.ca[k] * pstride + col;
    const float2* B = hb + item * bbs + (size_t)plan.cb[k] * pstride + col;
    float2* O = Q + item * qbs + (size_t)k * pstride + col;
    const int pl = col_pitch(f.n(), tx);
    f.template run_io<true>(
        smem + c * pl, t, true,
        [&](int y) {
            return okc ? cmulc(__ldg(&A[(size_t)y * WP]), __ldg(&B[(size_t)y * WP])) : make_float2(0.f, 0.f);
        },
        [&](int y, float2 v) {
            if (okc) O[(size_t)y * WP] = v;
        });
}

// ── inverse rows ────────────────────────────────────────────────────────────────────────────

// Task (row y, correlation pair (2p, 2p + 1)) of item blockIdx.y: Z = Q1 + i·Q2 on the row's half
// spectrum, conj(Q1) + i·conj(Q2) mirrored above it, its inverse FFT the two real rows, written
// over Q1's and Q2's row (a row of WP complex holds the nx reals). The task's lines are in one
// block and every line reads its inputs before the block's first barrier and writes after it, so
// writing in place is safe. Blocks of few lines, 1024 threads of them per SM: a line's barriers then hold
// up no more than its block, and the others' loads go on (two blocks of 512, then four of 256, then
// kRowT: 4096² rows and score of 18 correlations 1405 → 1281 µs, 104 sweep maps of 192² 453 → 409 →
// 333). S = 2: two lines of nx/2 points per task, line s the outputs
// x ≡ s (mod 2) after one decimation-in-frequency step.
template <class F, int S>
__global__ void __launch_bounds__(F::kRowT, 1024 / F::kRowT) k_inv_rows(float2* __restrict__ Q, size_t pstride, int WP, int nx, int ntask,
                                                     int n_corr, F f, int lpb, const float2* __restrict__ tw_nx,
                                                     size_t qbs) {
    extern __shared__ float2 smem[];
    Q += (size_t)blockIdx.y * qbs;
    const int L = f.n(), tl = f.tl(), npairs = (n_corr + 1) / 2;
    const int line = threadIdx.x / tl, t = threadIdx.x - line * tl;
    const int task = blockIdx.x * (lpb / S) + line / S, s = line % S;
    const bool act = line < lpb && task < ntask;
    const int y = act ? task / npairs : 0, k1 = act ? 2 * (task - y * npairs) : 0;
    const bool has2 = k1 + 1 < n_corr;
    float2* q1 = Q + (size_t)k1 * pstride + (size_t)y * WP;
    float2* q2 = has2 ? q1 + pstride : q1;
    float *o1 = reinterpret_cast<float*>(q1), *o2 = reinterpret_cast<float*>(q2);
    auto full = [&](int x) {
        const int ix = (x <= nx / 2) ? x : nx - x;
        const float2 a = q1[ix];
        const float2 b = has2 ? q2[ix] : make_float2(0.f, 0.f);
        return (x <= nx / 2) ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, b.x - a.y);
    };
    f.template run_io<true>(
        smem + (line < lpb ? line : 0) * padded_len(L), t, act,
        [&](int m) {
            if constexpr (S == 1) {
                return full(m);
            } else {
                const float2 lo = full(m), hi = full(m + L);
                if (s == 0) return cadd(lo, hi);
                return cmul(cadd(lo, cmul(hi, cconj(__ldg(&tw_nx[L])))), cconj(__ldg(&tw_nx[m])));
            }
        },
        [&](int m, float2 z) {
            o1[m * S + s] = z.x;
            if (has2) o2[m * S + s] = z.y;
        });
}

inline int lines_per_block(int tl, int want_threads) { return std::max(1, want_threads / tl); }
// column tile of a runtime line: as many lines as maxt threads hold (no more than the columns), within
// the shared memory of 1024 / maxt blocks per SM; whole 32-byte sectors (4 columns) where it can be
inline int col_tile(int n, int tl, int ncols, int maxt) {
    int tx = std::min(lines_per_block(tl, maxt), ncols);
    const size_t room = (maxt > 512 ? 220 : 110) * 1024;
    while (tx > 1 && (size_t)tx * col_pitch(n, tx) * sizeof(float2) > room) tx >>= 1;
    if (tl > 16) return tx >= 4 ? tx / 4 * 4 : tx;
    // short lines in wide tiles: the same number of tiles, balanced, no last tile of mostly idle columns
    const int tiles = (ncols + tx - 1) / tx;
    return (ncols + tiles - 1) / tiles;
}

// Blocks per SM the column kernels of a compile-time line are compiled for. The passes wait on their
// loads (2 to 4 blocks of 64-register threads left the schedulers 66 % idle), so the blocks are small
// (kTx columns) and take the registers that 1152 (forward) or 1280 threads (inverse) per SM leave, 56 or
// 48 for the 16 points of a thread; 1536 threads (40 registers) spill, except where a thread holds 9
// points at most (col_inv_tl). Longer lines: two blocks while that is 48 registers (2304 points: 491 →
// 302 µs; the forward pass of 2592 lost 15 %), else one. Inverse columns of 104 sweep maps of 192²:
// 600 → 351 µs, 256²: 590 → 390; of a map of 864²: 55 → 49, 1536²: 172 → 136.
template <class F>
__host__ __device__ constexpr int col_blocks(bool inverse) {
    constexpr int T = F::kTx * F::kTl;
    if (T == 0 || T > (inverse ? 720 : 640)) return 1;
    if (T > 512) return 2;
    const int want = !inverse ? 1152 : F::kOne ? 1536 : 1280;
    return want / T > 0 ? want / T : 1;
}

template <class F, Pass P, int MAXT, int MINB>
cudaError_t launch_cols(F f, const PassArgs& a, cudaStream_t st) {
    const MapGeom& g = a.g;
    const size_t pstride = (size_t)g.ny * g.WP;
    const int tl = f.tl(), ncols = g.nx / 2 + 1, tx = F::kTx ? F::kTx : col_tile(g.ny, tl, ncols, MAXT);
    // short lines: the planes' columns laid end to end, each plane's rounded up to whole sectors (97
    // columns in tiles of 16 would leave 13 % of the threads idle)
    const int npad = F::kTx && tl <= 32 ? (ncols + 3) / 4 * 4 : 0, tiles = (ncols + tx - 1) / tx;
    const size_t sm = (size_t)tx * col_pitch(g.ny, tx) * sizeof(float2);
    cudaError_t e;
    if constexpr (P == Pass::FwdCols) {
        const int planes = a.plan->n_real * a.batch;
        auto k = 2 * g.ch <= g.ny ? k_cols<F, false, true, MAXT, MINB> : k_cols<F, false, false, MAXT, MINB>;
        if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) != cudaSuccess) return e;
        const dim3 grid = npad ? dim3((planes * npad + tx - 1) / tx) : dim3(tiles, planes);
        k<<<grid, tx * tl, sm, st>>>(a.half, pstride, g.WP, ncols, npad, planes, g.ch, f, tx);
    } else {
        auto k = k_inv_cols<F, MAXT, MINB>;
        if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) != cudaSuccess) return e;
        const dim3 grid = npad ? dim3((a.plan->n_corr * npad + tx - 1) / tx, 1, a.batch) : dim3(a.plan->n_corr, tiles, a.batch);
        k<<<grid, tx * tl, sm, st>>>(a.half, a.half_b, pstride, g.WP, ncols, npad, *a.plan, f, tx, a.Q, a.half_stride,
                                     a.b_stride, a.q_stride);
    }
    return cudaGetLastError();
}
template <Pass P, class F>
cudaError_t run_cols(F f, const PassArgs& a, cudaStream_t st) {
    if constexpr (F::kTx != 0) {
        constexpr int T = F::kTx * F::kTl, B = col_blocks<F>(P == Pass::InvCols);
        return launch_cols<F, P, (B > 1 || T <= 512 ? T : 1024), B>(f, a, st);
    } else {
        // 512 threads, two blocks per SM, while 4 lines (a 32-byte sector of columns) fit
        return 4 * f.tl() <= 512 ? launch_cols<F, P, 512, 2>(f, a, st) : launch_cols<F, P, 1024, 1>(f, a, st);
    }
}

template <class F>
cudaError_t run_rows(F f, const PassArgs& a, cudaStream_t st) {
    const MapGeom& g = a.g;
    const CorrPlanDev& plan = *a.plan;
    const size_t pstride = (size_t)g.ny * g.WP;
    const int tl = f.tl();
    cudaError_t e;
    // rows: whole tasks (S lines) per block of up to kRowT threads
    if (a.S != 1 && a.S != 2) return cudaErrorInvalidConfiguration;
    const int lpb = std::max(a.S, lines_per_block(tl, F::kRowT) / a.S * a.S), ntask = g.ny * ((plan.n_corr + 1) / 2);
    if (lpb * tl > F::kRowT) return cudaErrorInvalidConfiguration;
    const size_t sm = (size_t)lpb * padded_len(f.n()) * sizeof(float2);
    auto k = a.S == 1 ? k_inv_rows<F, 1> : k_inv_rows<F, 2>;
    if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) != cudaSuccess) return e;
    k<<<dim3((ntask + lpb / a.S - 1) / (lpb / a.S), a.batch), lpb * tl, sm, st>>>(a.Q, pstride, g.WP, g.nx, ntask, plan.n_corr,
                                                                                  f, lpb, a.tw_nx, a.q_stride);
    return cudaGetLastError();
}

// One pass over a batch with line policy F.
template <class F>
cudaError_t run_pass(Pass p, F f, const PassArgs& a, cudaStream_t st) {
    const MapGeom& g = a.g;
    const CorrPlanDev& plan = *a.plan;
    const size_t pstride = (size_t)g.ny * g.WP;
    const int tl = f.tl();
    cudaError_t e;
    if (p == Pass::FwdRows) {
        const int n_cplx = (plan.n_real + 1) / 2;
        // The row's 3 lines at once (5 planes) where 512 threads hold them, else up to 256 threads of its 8.
        // Lines of whole warps, two or more of them: as many as 128 threads hold, one at least; the row's
        // others follow, and other rows' blocks fill the barriers (two sides of a map of 2048²: 98 → 76 µs,
        // 1536²: 90 → 77, 1024²: 28 → 25; 72 and 81 threads a line lost up to a third).
        const int lines = std::min(n_cplx, tl >= 64 && tl % 32 == 0          ? lines_per_block(tl, 128)
                                           : n_cplx <= 3 && n_cplx * tl <= 512 ? n_cplx
                                                                               : lines_per_block(tl, 256));
        const int products = plan.planes[plan.n_real - 1] >= 5;
        auto smem = [&](int rows) { return (size_t)lines * padded_len(g.nx) * sizeof(float2) + (size_t)rows * g.cw * sizeof(float); };
        size_t sm = smem(products ? 9 : 5);
        auto k = 2 * g.cw <= g.nx ? k_fwd_rows<F, true, false> : k_fwd_rows<F, false, false>;
        // A roto-scale grid has as many cells to a row as the line has points: from 5832 points on, nine rows
        // of them and the line do not fit shared memory, six do up to 6912.
        if constexpr (F::kLong) {
            if (products && 2 * g.cw > g.nx && sm > kRowShared) {
                sm = smem(6);
                k = k_fwd_rows<F, false, true>;
            }
        }
        if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) != cudaSuccess) return e;
        k<<<dim3(g.ch, a.batch), lines * tl, sm, st>>>(a.grid, g.cw, g.ch, g.WP, plan, f, lines, products, a.half,
                                                       pstride, a.grid_stride, a.half_stride);
        return cudaGetLastError();
    }
    if (p == Pass::FwdCols) return run_cols<Pass::FwdCols>(f, a, st);
    if (p == Pass::InvCols) return run_cols<Pass::InvCols>(f.inv(), a, st);
    return run_rows(f.row(), a, st);
}

}  // namespace

// the translation units that instantiate the compile-time lines (lines_*.cu); each returns false for lengths it does not carry
bool pass_lines_0(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e);
bool pass_lines_1(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e);
bool pass_lines_2(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e);
bool pass_lines_3(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e);
bool pass_lines_4(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e);
bool pass_lines_5(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e);
bool pass_lines_6(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e);
bool pass_lines_7(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e);

}  // namespace zc
