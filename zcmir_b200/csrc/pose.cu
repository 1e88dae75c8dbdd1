// Pose scores and gradients on the GPU: the 45 overlap moment sums of many poses at once, the
// score and its gradient coefficients (float64), and the tangent gradient with the Gauss–Newton
// matrix. Restated from the reference's shaders/smi.wgsl (overlap_moments 977-1057, taper
// 336-351, boundary_value 353-366, score_dva 1059-1081, tangent_grad 1123-1272) and
// src/moments.zig (scoreFromMoments 91-172).
//
// One direction warps image a (moving) onto image b (fixed): every b pixel x samples a's
// features bilinearly at H⁻¹(x + 1) − 1, weighted by a 2-px ramp inside a's valid border. Blocks
// of pose p sum their pixels in float32 per thread, then float64 across the block; the pose's
// blocks' totals are added in block order by the last of them to finish (block_add). One launch
// takes both directions of every pose; its last block per pose and direction also scores it, so a
// pose score is one kernel and its result (with out.host) is written to the caller's page-locked
// memory by that block: a score of a 256² pair took 88 µs as two moment launches, a one-thread
// score kernel and four copies.
#include <array>
#include <atomic>
#include <algorithm>

#include "common.cuh"
#include "kernels.hpp"

namespace zc {
namespace {

constexpr float kTaper = 2.0f;
constexpr int kMom = 45, kCoef = 102, kG0 = 40, kQ0 = 85, kGrad = 44;

__device__ __forceinline__ int tri4(int i, int j) {
    const int a = min(i, j), b = max(i, j);
    return a * 4 - (a * (a + 1)) / 2 + b;
}

// The block's k ≤ 48 float64 totals (thread t < k holds total t; the others pass anything) added
// into out[0 .. k) of the launch's row `row` (a pose in one direction) of nblk blocks. With r.part: every block
// stores its totals at part[(row · cap + block) · k], cap the grid's blocks per row, then the row's
// last block to finish (the old value of its ticket is nblk − 1) adds them in a fixed order — group
// g of ⌊256 / k⌋ threads takes blocks g, g + groups, …, and thread t adds the groups' totals 0, 1, …
// — puts the ticket back to 0 and returns true with the totals in tot. Every thread of the block
// calls it. Without r.part: float64 atomics, and false.
__device__ bool block_add(double s, int k, double* __restrict__ out, const PoseRed& r, int row, int nblk, double* tot) {
    const int t = threadIdx.x;
    if (!r.part) {
        if (t < k) atomicAdd(&out[t], s);
        return false;
    }
    __shared__ int last;
    __shared__ double grp[8][48];
    double* part = r.part + (size_t)row * gridDim.x * k;
    if (t < k) part[(size_t)blockIdx.x * k + t] = s;
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(&r.ticket[row], 1u) == (unsigned)(nblk - 1);
    __syncthreads();
    if (!last) return false;  // uniform over the block
    __threadfence();
    const int ng = min((int)blockDim.x / k, 8), g = t / k, e = t - g * k;
    if (g < ng) {
        double a = 0.0;
#pragma unroll 8
        for (int b = g; b < nblk; b += ng) a += __ldcg(&part[(size_t)b * k + e]);
        grp[g][e] = a;
    }
    __syncthreads();
    if (t < k) {
        double a = 0.0;
        for (int q = 0; q < ng; ++q) a += grp[q][t];
        out[t] = tot[t] = a;
    }
    if (t == 0) r.ticket[row] = 0;
    __syncthreads();
    return true;
}

// The warp's sums of 48 values per lane: each step adds and halves the values a lane still carries
// (48 shuffles, not 240). Lane l is left with values warp_first(l) .. + 2 in v[0..2] (lanes l and
// l ^ 1 hold the same).
__device__ __forceinline__ void warp_sums48(float (&v)[48]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 24, bit = 16; n >= 3; n >>= 1, bit >>= 1)
#pragma unroll
        for (int i = 0; i < 24; ++i) {
            if (i >= n) continue;
            const bool up = (lane & bit) != 0;
            const float other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[n + i], bit);
            v[i] = (up ? v[n + i] : v[i]) + other;
        }
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 1);
}
__device__ __forceinline__ int warp_first(int lane) {
    return ((lane >> 4) & 1) * 24 + ((lane >> 3) & 1) * 12 + ((lane >> 2) & 1) * 6 + ((lane >> 1) & 1) * 3;
}

// what a pose launch reads and writes; direction d samples image d at every pixel of image 1 − d
struct PoseLaunch {
    const float4* f[2];
    int w[2], h[2];
    int n;                 // poses of the call
    int p0;                // the launch's first: poses p0 .. p0 + gridDim.y − 1
    int nblk[2];           // blocks per pose of each direction
    const float* hinv;     // inverse poses, a row each: direction 0's n, then direction 1's
    PoseFfd ffd[2];
    const unsigned char* mask;
    PoseRed rd;
    double* out;           // rows of totals, direction 0's n then direction 1's
    double* host;          // the same in page-locked memory (nullable)
    // moments: the score of each row (scored), its coefficients; tangent: coefficients, generators
    int scored, exact, hess;
    float* coef;
    double *score, *host_score;
    float gens[144];
    int n_inl;             // rows of inl in place of hinv (0: none)
    float inl[9 * kPoseInline];
};

__device__ __forceinline__ float hinv_at(const PoseLaunch& L, int row, int e) {
    return L.n_inl ? L.inl[row * 9 + e] : L.hinv[(size_t)row * 9 + e];
}

// (w, ∂w/∂fx, ∂w/∂fy) of the border taper at (fx, fy) in a w×h image
__device__ __forceinline__ void taper(float fx, float fy, float w, float h, float& t, float& tx, float& ty) {
    auto ramp = [](float v, float lo, float hi, float& val, float& dv) {
        const float a = (v - lo) / kTaper, b = (hi - v) / kTaper;
        const float ca = fminf(fmaxf(a, 0.f), 1.f), cb = fminf(fmaxf(b, 0.f), 1.f);
        const float da = (a > 0.f && a < 1.f) ? 1.f / kTaper : 0.f;
        const float db = (b > 0.f && b < 1.f) ? -1.f / kTaper : 0.f;
        val = ca * cb;
        dv = da * cb + ca * db;
    };
    float vx, dx, vy, dy;
    ramp(fx, 2.f, w - 3.f, vx, dx);
    ramp(fy, 2.f, h - 3.f, vy, dy);
    t = vx * vy;
    tx = dx * vy;
    ty = vx * dy;
}

// ── the B-spline (smi.wgsl:198-240 cubic_w, dest_half, ffd_disp) ──

constexpr int kFfdMax = 16;  // lattice side (src/pose.zig:17 FFD_MAX)

__device__ __forceinline__ float4 cubic_w(float t) {
    const float t2 = t * t, t3 = t2 * t;
    return make_float4((1.f - t) * (1.f - t) * (1.f - t) / 6.f, (3.f * t3 - 6.f * t2 + 4.f) / 6.f,
                       (-3.f * t3 + 3.f * t2 + 3.f * t + 1.f) / 6.f, t3 / 6.f);
}
__device__ __forceinline__ float comp4(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// The 2×2 taps at i00, i00 + 1, i00 + aw, i00 + aw + 1 of an image whose four feature planes are
// interleaved (one float4 per pixel): one 16-byte load per tap instead of one per plane and tap.
struct Taps4 {
    float4 v00, v10, v01, v11;
};
__device__ __forceinline__ Taps4 taps4(const float4* __restrict__ a, size_t i00, int aw) {
    return {__ldg(&a[i00]), __ldg(&a[i00 + 1]), __ldg(&a[i00 + aw]), __ldg(&a[i00 + aw + 1])};
}

// A block's view of a spline: its control points staged in shared memory (c null: none).
struct FfdView {
    const float* c;
    int g, source;
};

// stage pose `pose`'s control points (all threads call it; a __syncthreads must follow)
__device__ __forceinline__ FfdView ffd_view(const PoseFfd& f, float* sh, int pose = 0) {
    if (!f.cps || f.g < 2) return FfdView{nullptr, 0, 0};
    const float* c = f.cps + (size_t)pose * f.stride;
    for (int i = threadIdx.x; i < 2 * f.g * f.g; i += blockDim.x) sh[i] = c[i];
    return FfdView{sh, f.g, f.source};
}

// the displacement (pixels) at the 0-based point (xf, yf) of the lattice's rw × rh image: 0
// outside it; half-image units scaled by (rw/2, rh/2); clamped lattice indices
__device__ __forceinline__ float2 ffd_disp(const FfdView& f, float xf, float yf, float rw, float rh) {
    if (xf < 0.f || yf < 0.f || xf > rw - 1.f || yf > rh - 1.f) return make_float2(0.f, 0.f);
    const int g = f.g;
    const float hx = fmaxf(rw, 1.f) * 0.5f, hy = fmaxf(rh, 1.f) * 0.5f;
    const float spx = fmaxf(rw - 1.f, 1.f) / (float)(g - 1), spy = fmaxf(rh - 1.f, 1.f) / (float)(g - 1);
    const float su = xf / spx, sv = yf / spy;
    const int iu = (int)floorf(su), iv = (int)floorf(sv);
    const float4 bu = cubic_w(fminf(fmaxf(su - (float)iu, 0.f), 1.f));
    const float4 bv = cubic_w(fminf(fmaxf(sv - (float)iv, 0.f), 1.f));
    float dx = 0.f, dy = 0.f;
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
        const int j = min(max(iv - 1 + jj, 0), g - 1);
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) {
            const int i = min(max(iu - 1 + ii, 0), g - 1);
            const float w = comp4(bu, ii) * comp4(bv, jj);
            const int o = (j * g + i) * 2;
            dx = dx + w * (f.c[o] * hx);
            dy = dy + w * (f.c[o + 1] * hy);
        }
    }
    return make_float2(dx, dy);
}

// A walk of a row's nblk blocks over a w × h image in tiles of 8 × 4 pixels, one tile per warp and
// step (lane → (lane mod 8, lane / 8)): a warp's 32 pixels are a compact patch, so the bilinear taps
// they gather on the other image under any rotation fall on few rows (few sectors per load).
// Tile coordinates are stepped along, not divided out per tile.
struct TileWalk {
    int T, nt, step, tx, ty, sx, sy, ntx, lx, ly, w, h;
    __device__ __forceinline__ TileWalk(int w_, int h_, int nblk) : w(w_), h(h_) {
        ntx = (w + 7) >> 3;
        nt = ntx * ((h + 3) >> 2);
        const int lane = threadIdx.x & 31;
        lx = lane & 7;
        ly = lane >> 3;
        T = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
        step = (int)((nblk * blockDim.x) >> 5);
        ty = T / ntx;
        tx = T - ty * ntx;
        sy = step / ntx;
        sx = step - sy * ntx;
    }
    __device__ __forceinline__ bool ok() const { return T < nt; }
    __device__ __forceinline__ void next() {
        T += step;
        tx += sx;
        ty += sy;
        if (tx >= ntx) {
            tx -= ntx;
            ++ty;
        }
    }
    __device__ __forceinline__ int x() const { return (tx << 3) + lx; }
    __device__ __forceinline__ int y() const { return (ty << 2) + ly; }
    __device__ __forceinline__ bool in() const { return x() < w && y() < h; }
};

// pose sample position of b pixel (x, y) (smi.wgsl overlap_moments 1003-1016): with a spline on
// b the pixel moves first, X = (x + 1 + dx, y + 1 + dy); on a the sample H⁻¹X − 1 moves after.
// ph = H⁻¹X, (Xx, Xy) = X. False when outside a's valid interior.
template <bool FFD>
__device__ __forceinline__ bool sample_pos(const float* Hi, const FfdView& f, int x, int y, int aw, int ah, int bw,
                                           int bh, float& fx, float& fy, float3& ph, float& Xx, float& Xy) {
    Xx = (float)x + 1.f;
    Xy = (float)y + 1.f;
    if (FFD && !f.source) {
        const float2 d = ffd_disp(f, (float)x, (float)y, (float)bw, (float)bh);
        Xx = (float)x + 1.f + d.x;
        Xy = (float)y + 1.f + d.y;
    }
    ph.x = Hi[0] * Xx + Hi[1] * Xy + Hi[2];
    ph.y = Hi[3] * Xx + Hi[4] * Xy + Hi[5];
    ph.z = Hi[6] * Xx + Hi[7] * Xy + Hi[8];
    if (fabsf(ph.z) < 1e-8f) return false;
    if (ph.z == 1.f) {  // affine poses: the division is exact, skip it
        fx = ph.x - 1.f;
        fy = ph.y - 1.f;
    } else {
        fx = ph.x / ph.z - 1.f;
        fy = ph.y / ph.z - 1.f;
    }
    if (FFD && f.source) {
        const float2 d = ffd_disp(f, fx, fy, (float)aw, (float)ah);
        fx = fx + d.x;
        fy = fy + d.y;
    }
    return !(fx < 2.f || fy < 2.f || fx > (float)aw - 3.f || fy > (float)ah - 3.f);
}

// scoreFromMoments (src/moments.zig:91-172) in float64 by one warp: the score of the 45 sums st
// (shared memory) and the 102 coefficients [W 0–15, μ_B 16–19, M̂ 20–35, μ_A 36–39, g = ∂S/∂sums
// 40–84, Q 85–100, flag] the tangent pass reads (zero when the overlap is under 12 or a whitening
// fails). Lane 16·h + 4·i + j holds entry (i, j) of the 4 × 4 matrices, half h side A's or B's
// Gram matrix: a thread of its own took 14 µs over the same steps.
__device__ __forceinline__ double lane_get(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

__device__ void score_warp(const double* st, int exact, double ridge, float* __restrict__ out, double* score,
                           double* host_score) {
    const int lane = threadIdx.x & 31, h = lane >> 4, base = h * 16, i = (lane >> 2) & 3, j = lane & 3;
    auto fail = [&] {
        for (int k = lane; k < kCoef; k += 32) out[k] = 0.f;
        if (lane == 0) {
            *score = 0.0;
            if (host_score) *host_score = 0.0;
        }
    };
    const double nn = st[0];
    if (!(nn >= 12.0)) return fail();
    const double mai = st[1 + i] / nn, maj = st[1 + j] / nn, mbi = st[5 + i] / nn, mbj = st[5 + j] / nn;
    const double C = st[9 + 4 * i + j] / nn - mai * mbj;
    // Σ_k a(i, k)·b(k, j), a in half ha and b in half hb; ta, tb: the factor transposed
    auto mm = [&](double a, int ha, bool ta, double b, int hb, bool tb) {
        double r = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            r += lane_get(a, 16 * ha + (ta ? 4 * k + i : 4 * i + k)) * lane_get(b, 16 * hb + (tb ? 4 * j + k : 4 * k + j));
        return r;
    };
    double W = C, MN = 0.0, phi;  // MN: M̂ in half 0, N̂ in half 1
    if (!exact) {
        phi = h == 0 ? C * C : 0.0;
    } else {
        const int t0 = h ? 35 : 25;
        double g = st[t0 + tri4(i, j)] / nn - (h ? mbi * mbj : mai * maj);
        double tr = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) tr += lane_get(g, base + 5 * k);
        if (i == j) g += ridge * fmax(tr / 4, 1e-12);
        // Cholesky by columns; il: the inverse diagonal
        double L = 0.0, il[4];
        bool ok = true;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double piv = lane_get(g, base + 5 * k);
            ok = ok && piv > 0.0;
            const double d = sqrt(piv);
            il[k] = 1.0 / d;
            const double lik = lane_get(g, base + 4 * i + k) * il[k], ljk = lane_get(g, base + 4 * j + k) * il[k];
            if (j == k) L = i == k ? d : (i > k ? lik : 0.0);
            if (i > k && j > k) g -= lik * ljk;
        }
        if (!__all_sync(0xffffffffu, ok)) return fail();
        // column j of the inverse: L y = e_j, Lᵀ x = y
        double y[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            double v = r == j ? 1.0 : 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double l = lane_get(L, base + 4 * r + k);
                if (k < r) v -= l * y[k];
            }
            y[r] = v * il[r];
        }
#pragma unroll
        for (int r = 3; r >= 0; --r) {
            double v = y[r];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double l = lane_get(L, base + 4 * k + r);
                if (k > r) v -= l * y[k];
            }
            y[r] = v * il[r];
        }
        const double Gi = i == 0 ? y[0] : i == 1 ? y[1] : i == 2 ? y[2] : y[3];
        W = mm(mm(Gi, 0, false, C, 0, false), 0, false, Gi, 1, false);
        phi = h == 0 ? W * C : 0.0;
        // M̂ = W Cᵀ G_A⁻¹ (half 0), N̂ = Wᵀ C G_B⁻¹ (half 1)
        const double u = mm(W, 0, false, C, 0, true), v = mm(W, 0, true, C, 0, false), x = h ? v : u;
        MN = mm(x, h, false, Gi, h, false);
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) t += lane_get(MN, base + 5 * k);
        if (i == j) MN += t * ridge / 4;
    }
    const double sc = nn * warp_sum(phi);
    if (!isfinite(sc)) return fail();
    // g: the feature sums' entries ga (half 0), gb (half 1), and the products'
    const double wt = lane_get(W, 16 * h + 4 * j + i);  // W(j, i)
    double gm = h ? -2 * wt * maj + 2 * MN * mbj : -2 * W * mbj + 2 * MN * maj;
    gm += __shfl_xor_sync(0xffffffffu, gm, 1);
    gm += __shfl_xor_sync(0xffffffffu, gm, 2);
    const double gp = -(i == j ? 1.0 : 2.0) * MN;
    double rest = 0.0;
    if (j == 0) rest += gm * st[(h ? 5 : 1) + i];
    if (h == 0) rest += 2 * W * st[9 + 4 * i + j];
    if (j >= i) rest += gp * st[(h ? 35 : 25) + tri4(i, j)];
    rest = warp_sum(rest);
    const double Q = exact ? MN : mm(C, 0, false, C, 0, true);
    if (h == 0) {
        out[4 * i + j] = (float)W;
        out[20 + 4 * i + j] = (float)MN;
        out[kG0 + 9 + 4 * i + j] = (float)(2 * W);
        out[kQ0 + 4 * i + j] = (float)Q;
    }
    if (j == 0) {
        out[h ? 16 + i : 36 + i] = (float)(h ? mbi : mai);
        out[kG0 + (h ? 5 : 1) + i] = (float)gm;
    }
    if (j >= i) out[kG0 + (h ? 35 : 25) + tri4(i, j)] = (float)gp;
    if (lane == 0) {
        out[kG0] = (float)((sc - rest) / nn);
        out[kCoef - 1] = 0.f;
        *score = sc;
        if (host_score) *host_score = sc;
    }
}

// A pixel's sample: its weight, the 2 × 2 taps' features and its own, two features to a register
// pair as they are loaded.
struct PoseSample {
    bool ok;
    float wt, ax, ay;
    ulonglong2 v00, v10, v01, v11, vb;
};

// The 45 sums: 0 Σw, 1–4 Σw a, 5–8 Σw b, 9–24 Σw a_i b_j, 25–34 / 35–44 upper triangles of
// Σw a aᵀ and Σw b bᵀ. grid: (blocks, poses, directions). Features (0, 1) and (2, 3) go through
// the interpolation and the products they meet in as pairs (f32x2), the others alone: 39
// multiply-add instructions a pixel, not 73. U pixels' taps are loaded before the first is added:
// 1 where the launch fills the GPU (bound by instructions, 60 % of the issue slots at 24 warps an
// SM), 4 where few blocks are in flight and each waits on its loads. The order of every sum, and so
// its bits, is the same for any U.
template <bool FFD, int U>
__global__ void __launch_bounds__(256, FFD ? 2 : U == 1 ? 3 : 1) k_pose_moments(const __grid_constant__ PoseLaunch L) {
    __shared__ float red[8][48];
    __shared__ float cps[2 * kFfdMax * kFfdMax];
    __shared__ double tot[48];
    const int pose = L.p0 + blockIdx.y, d = blockIdx.z, row = d * L.n + pose, nblk = L.nblk[d];
    if ((int)blockIdx.x >= nblk || (L.mask && !L.mask[pose])) return;  // a masked pose's sums are read by nobody
    const float4 *__restrict__ fa = L.f[d], *__restrict__ fb = L.f[1 - d];
    const int aw = L.w[d], ah = L.h[d], bw = L.w[1 - d], bh = L.h[1 - d];
    const FfdView fv = ffd_view(L.ffd[d], cps, pose);
    float Hi[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) Hi[i] = hinv_at(L, row, i);
    if (FFD) __syncthreads();
    const float xhi = (float)aw - 3.f, yhi = (float)ah - 3.f;
    float n = 0.f;
    // a_i b_j as pairs (00,11) (02,13) (20,31) (22,33) and 01 10 03 12 21 30 23 32; a aᵀ and b bᵀ as
    // (00,11) (02,13) (22,33) and 01 03 12 23
    f32x2 sa[2] = {0, 0}, sb[2] = {0, 0}, ab[4] = {0, 0, 0, 0}, aa[3] = {0, 0, 0}, bb[3] = {0, 0, 0};
    float ab1[8] = {0, 0, 0, 0, 0, 0, 0, 0}, aa1[4] = {0, 0, 0, 0}, bb1[4] = {0, 0, 0, 0};
    TileWalk pw(bw, bh, nblk);
    while (pw.ok()) {
        PoseSample q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            q[u].ok = false;
            if (pw.ok() && pw.in()) {
                const int y = pw.y(), x = pw.x();
                float fx, fy, Xx, Xy;
                float3 ph;
                if (sample_pos<FFD>(Hi, fv, x, y, aw, ah, bw, bh, fx, fy, ph, Xx, Xy)) {
                    // the 2-px ramps: (v − 2) / 2 and (hi − v) / 2 clamped to [0, 1]
                    const float wt = __saturatef(fmaf(fx, 0.5f, -1.f)) * __saturatef((xhi - fx) * 0.5f) *
                                     (__saturatef(fmaf(fy, 0.5f, -1.f)) * __saturatef((yhi - fy) * 0.5f));
                    if (wt > 0.f) {
                        const float flx = floorf(fx), fly = floorf(fy);
                        q[u].ok = true, q[u].wt = wt, q[u].ax = fx - flx, q[u].ay = fy - fly;
                        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(fa) + ((int)fly * aw + (int)flx);  // fx, fy ≥ 2
                        q[u].v00 = __ldg(p), q[u].v10 = __ldg(p + 1), q[u].v01 = __ldg(p + aw), q[u].v11 = __ldg(p + aw + 1);
                        q[u].vb = __ldg(reinterpret_cast<const ulonglong2*>(fb) + (y * bw + x));
                    }
                }
            }
            if (U > 1 || u == 0) pw.next();
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!q[u].ok) continue;
            const PoseSample& s = q[u];
            const f32x2 x1 = pack2(s.ax, s.ax), x0 = pack2(1.f - s.ax, 1.f - s.ax);
            const f32x2 y1 = pack2(s.ay, s.ay), y0 = pack2(1.f - s.ay, 1.f - s.ay), w2 = pack2(s.wt, s.wt);
            const f32x2 a01 = fma2(fma2(s.v00.x, x0, mul2(s.v10.x, x1)), y0, mul2(fma2(s.v01.x, x0, mul2(s.v11.x, x1)), y1));
            const f32x2 a23 = fma2(fma2(s.v00.y, x0, mul2(s.v10.y, x1)), y0, mul2(fma2(s.v01.y, x0, mul2(s.v11.y, x1)), y1));
            const f32x2 b01 = s.vb.x, b23 = s.vb.y;
            const f32x2 wa01 = mul2(a01, w2), wa23 = mul2(a23, w2), wb01 = mul2(b01, w2), wb23 = mul2(b23, w2);
            float a0, a1, a2, a3, b0, b1, b2, b3, wa0, wa1, wa2, wa3, wb0, wb1, wb2, wb3;
            unpack2(a01, a0, a1), unpack2(a23, a2, a3), unpack2(b01, b0, b1), unpack2(b23, b2, b3);
            unpack2(wa01, wa0, wa1), unpack2(wa23, wa2, wa3), unpack2(wb01, wb0, wb1), unpack2(wb23, wb2, wb3);
            n += s.wt;
            sa[0] = add2(sa[0], wa01), sa[1] = add2(sa[1], wa23);
            sb[0] = add2(sb[0], wb01), sb[1] = add2(sb[1], wb23);
            ab[0] = fma2(wa01, b01, ab[0]), ab[1] = fma2(wa01, b23, ab[1]);
            ab[2] = fma2(wa23, b01, ab[2]), ab[3] = fma2(wa23, b23, ab[3]);
            ab1[0] = fmaf(wa0, b1, ab1[0]), ab1[1] = fmaf(wa1, b0, ab1[1]), ab1[2] = fmaf(wa0, b3, ab1[2]);
            ab1[3] = fmaf(wa1, b2, ab1[3]), ab1[4] = fmaf(wa2, b1, ab1[4]), ab1[5] = fmaf(wa3, b0, ab1[5]);
            ab1[6] = fmaf(wa2, b3, ab1[6]), ab1[7] = fmaf(wa3, b2, ab1[7]);
            aa[0] = fma2(wa01, a01, aa[0]), aa[1] = fma2(wa01, a23, aa[1]), aa[2] = fma2(wa23, a23, aa[2]);
            aa1[0] = fmaf(wa0, a1, aa1[0]), aa1[1] = fmaf(wa0, a3, aa1[1]), aa1[2] = fmaf(wa1, a2, aa1[2]);
            aa1[3] = fmaf(wa2, a3, aa1[3]);
            bb[0] = fma2(wb01, b01, bb[0]), bb[1] = fma2(wb01, b23, bb[1]), bb[2] = fma2(wb23, b23, bb[2]);
            bb1[0] = fmaf(wb0, b1, bb1[0]), bb1[1] = fmaf(wb0, b3, bb1[1]), bb1[2] = fmaf(wb1, b2, bb1[2]);
            bb1[3] = fmaf(wb2, b3, bb1[3]);
        }
    }
    float v[48];
    v[0] = n, v[45] = v[46] = v[47] = 0.f;
    unpack2(sa[0], v[1], v[2]), unpack2(sa[1], v[3], v[4]);
    unpack2(sb[0], v[5], v[6]), unpack2(sb[1], v[7], v[8]);
    unpack2(ab[0], v[9], v[14]), unpack2(ab[1], v[11], v[16]), unpack2(ab[2], v[17], v[22]), unpack2(ab[3], v[19], v[24]);
    v[10] = ab1[0], v[13] = ab1[1], v[12] = ab1[2], v[15] = ab1[3];
    v[18] = ab1[4], v[21] = ab1[5], v[20] = ab1[6], v[23] = ab1[7];
    auto tri = [&](const f32x2(&q)[3], const float(&r)[4], int o) {
        unpack2(q[0], v[o], v[o + 4]), unpack2(q[1], v[o + 2], v[o + 6]), unpack2(q[2], v[o + 7], v[o + 9]);
        v[o + 1] = r[0], v[o + 3] = r[1], v[o + 5] = r[2], v[o + 8] = r[3];
    };
    tri(aa, aa1, 25), tri(bb, bb1, 35);
    warp_sums48(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if ((lane & 1) == 0)
#pragma unroll
        for (int i = 0; i < 3; ++i) red[w][warp_first(lane) + i] = v[i];
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < kMom)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += (double)red[i][threadIdx.x];
    if (!block_add(s, kMom, L.out + (size_t)row * kMom, L.rd, d * gridDim.y + blockIdx.y, nblk, tot)) return;
    if (L.host && threadIdx.x < kMom) L.host[(size_t)row * kMom + threadIdx.x] = tot[threadIdx.x];
    if (L.scored && threadIdx.x < 32)
        score_warp(tot, L.exact, 1e-4, L.coef + (size_t)row * kCoef, L.score + row, L.host_score ? L.host_score + row : nullptr);
}

// the scores and coefficients of n poses' sums, a warp each
__global__ void __launch_bounds__(128) k_pose_coefs(const double* __restrict__ sums, int n, int exact, double ridge,
                                                    float* __restrict__ coef, double* __restrict__ score) {
    __shared__ double st[4][kMom];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, pose = blockIdx.x * 4 + w;
    if (pose >= n) return;
    for (int k = lane; k < kMom; k += 32) st[w][k] = sums[(size_t)pose * kMom + k];
    __syncwarp();
    score_warp(st[w], exact, ridge, coef + (size_t)pose * kCoef, score + pose, nullptr);
}

// The gradient over the tangent coordinates and (hess) the Gauss–Newton matrix Σ wt·J_aᵀ Q J_a:
// per pose 44 sums (8 gradient, then the 8×8 upper triangle row by row). Per pixel the gradient
// needs the two scalars cx, cy = (∂S/∂v_a)·∇v_a plus the taper's boundary term, times each
// tangent's flow ∂(sample)/∂ξ_k = ((M_k X)·ph.z − ph·(M_k X).z)/ph.z², M_k = −H⁻¹ G_k.
template <bool FFD>
__global__ void __launch_bounds__(256) k_pose_tangent(const __grid_constant__ PoseLaunch L) {
    __shared__ float Hs[9], Mk[8][9], cf[kCoef];
    __shared__ float red[8][48];
    __shared__ float cps[2 * kFfdMax * kFfdMax];
    __shared__ double tot[48];
    const int pose = L.p0 + blockIdx.y, d = blockIdx.z, row = d * L.n + pose, nblk = L.nblk[d], hess = L.hess;
    if ((int)blockIdx.x >= nblk || (L.mask && !L.mask[pose])) return;  // a masked pose's sums are read by nobody
    const float4 *__restrict__ fa = L.f[d], *__restrict__ fb = L.f[1 - d];
    const int aw = L.w[d], ah = L.h[d], bw = L.w[1 - d], bh = L.h[1 - d];
    if (threadIdx.x < 9) Hs[threadIdx.x] = hinv_at(L, row, threadIdx.x);
    for (int k = threadIdx.x; k < kCoef; k += blockDim.x) cf[k] = L.coef[(size_t)row * kCoef + k];
    const FfdView fv = ffd_view(L.ffd[d], cps, pose);
    __syncthreads();
    if (threadIdx.x < 72) {
        const int k = threadIdx.x / 9, e = threadIdx.x % 9, r = e / 3, c = e % 3;
        const float* G = L.gens + 72 * d + k * 9;
        Mk[k][e] = -(Hs[r * 3] * G[c] + Hs[r * 3 + 1] * G[3 + c] + Hs[r * 3 + 2] * G[6 + c]);
    }
    __syncthreads();
    float Hi[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) Hi[i] = Hs[i];
    float g8[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    float h36[36];
#pragma unroll
    for (int k = 0; k < 36; ++k) h36[k] = 0.f;
    for (TileWalk pw(bw, bh, nblk); pw.ok(); pw.next()) {
        if (!pw.in()) continue;
        const int y = pw.y(), x = pw.x();
        const size_t t = (size_t)y * bw + x;
        float fx, fy, X, Y;
        float3 ph;
        if (!sample_pos<FFD>(Hi, fv, x, y, aw, ah, bw, bh, fx, fy, ph, X, Y)) continue;
        float wt, tpx, tpy;
        taper(fx, fy, (float)aw, (float)ah, wt, tpx, tpy);
        const float flx = floorf(fx), fly = floorf(fy);
        const float ax = fx - flx, ay = fy - fly;
        const size_t i00 = (size_t)(int)fly * aw + (int)flx;  // fx, fy ≥ 2 here
        float va[4], gx[4], gy[4], vb[4];
        const Taps4 tp = taps4(fa, i00, aw);
        const float4 b4 = __ldg(&fb[t]);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const float v00 = comp4(tp.v00, p), v10 = comp4(tp.v10, p);
            const float v01 = comp4(tp.v01, p), v11 = comp4(tp.v11, p);
            va[p] = (v00 * (1.f - ax) + v10 * ax) * (1.f - ay) + (v01 * (1.f - ax) + v11 * ax) * ay;
            gx[p] = (v10 - v00) * (1.f - ay) + (v11 - v01) * ay;
            gy[p] = (v01 - v00) * (1.f - ax) + (v11 - v10) * ax;
            vb[p] = comp4(b4, p);
        }
        // ∂S/∂v_a = 2 (W (v_b − μ_B) − M̂ (v_a − μ_A))
        float ra[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            float s = 0.f;
#pragma unroll
            for (int b = 0; b < 4; ++b) s += cf[a * 4 + b] * (vb[b] - cf[16 + b]) - cf[20 + a * 4 + b] * (va[b] - cf[36 + b]);
            ra[a] = 2.f * s;
        }
        // the taper's boundary term: Σ_k g_k φ_k(v_a, v_b)
        float bwv = 0.f;
        if (tpx != 0.f || tpy != 0.f) {
            const float* g = cf + kG0;
            float s = g[0];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s += g[1 + i] * va[i] + g[5 + i] * vb[i];
#pragma unroll
                for (int j = 0; j < 4; ++j) s += g[9 + i * 4 + j] * va[i] * vb[j];
#pragma unroll
                for (int j = i; j < 4; ++j) s += g[25 + tri4(i, j)] * va[i] * va[j] + g[35 + tri4(i, j)] * vb[i] * vb[j];
            }
            bwv = s;
        }
        float dga = 0.f, dgb = 0.f;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            dga += ra[p] * gx[p];
            dgb += ra[p] * gy[p];
        }
        const float cx = wt * dga + bwv * tpx, cy = wt * dgb + bwv * tpy;
        const float iz2 = 1.f / fmaxf(ph.z * ph.z, 1e-12f);
        float px[8], py[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float* M = Mk[k];
            const float wx = M[0] * X + M[1] * Y + M[2];
            const float wy = M[3] * X + M[4] * Y + M[5];
            const float wz = M[6] * X + M[7] * Y + M[8];
            px[k] = (wx * ph.z - ph.x * wz) * iz2;
            py[k] = (wy * ph.z - ph.y * wz) * iz2;
            g8[k] += cx * px[k] + cy * py[k];
        }
        if (hess) {
            float qgx[4], qgy[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                float sx = 0.f, sy = 0.f;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    sx += cf[kQ0 + a * 4 + b] * gx[b];
                    sy += cf[kQ0 + a * 4 + b] * gy[b];
                }
                qgx[a] = sx;
                qgy[a] = sy;
            }
            float sxx = 0.f, sxy = 0.f, syx = 0.f, syy = 0.f;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                sxx += gx[a] * qgx[a];
                sxy += gx[a] * qgy[a];
                syx += gy[a] * qgx[a];
                syy += gy[a] * qgy[a];
            }
            int h = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float rk = wt * (sxx * px[k] + syx * py[k]);
                const float sk = wt * (sxy * px[k] + syy * py[k]);
#pragma unroll
                for (int l = k; l < 8; ++l) h36[h++] += rk * px[l] + sk * py[l];
            }
        }
    }
    float v[48];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = g8[k];
#pragma unroll
    for (int k = 0; k < 40; ++k) v[8 + k] = k < 36 ? h36[k < 36 ? k : 0] : 0.f;
    warp_sums48(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if ((lane & 1) == 0)
#pragma unroll
        for (int i = 0; i < 3; ++i) red[w][warp_first(lane) + i] = v[i];
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < kGrad)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += (double)red[i][threadIdx.x];
    if (!block_add(s, kGrad, L.out + (size_t)row * kGrad, L.rd, d * gridDim.y + blockIdx.y, nblk, tot)) return;
    if (L.host && threadIdx.x < kGrad) L.host[(size_t)row * kGrad + threadIdx.x] = tot[threadIdx.x];
}

// ∂score/∂(control points cp0 .. cp0 + 15) of pose 0 (smi.wgsl ffd_grad 1275-1417): per valid
// pixel the two scalars Gx, Gy — (∂S/∂v_a)·∇v_a and the taper's boundary term along the sample's
// motion under a unit x or y displacement of one control point (through H⁻¹ on a b lattice,
// directly on an a lattice), per unit basis weight — then each control point of the chunk takes
// its basis weight B_i(u) B_j(v) (clamped lattice indices summed) times them.
__global__ void __launch_bounds__(256) k_pose_ffd_grad(const float4* __restrict__ fa, int aw, int ah,
                                                       const float4* __restrict__ fb, int bw, int bh,
                                                       const float* __restrict__ hinv, const float* __restrict__ coef,
                                                       PoseFfd ffd, int cp0, double* __restrict__ out, PoseRed rd) {
    __shared__ float Hs[9], cf[kCoef];
    __shared__ float red[8][32];
    __shared__ float cps[2 * kFfdMax * kFfdMax];
    if (threadIdx.x < 9) Hs[threadIdx.x] = hinv[threadIdx.x];
    for (int k = threadIdx.x; k < kCoef; k += blockDim.x) cf[k] = coef[k];
    const FfdView fv = ffd_view(ffd, cps);
    __syncthreads();
    float Hi[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) Hi[i] = Hs[i];
    const int g = fv.g;
    const bool src = fv.source != 0;
    const float lw = src ? (float)aw : (float)bw, lh = src ? (float)ah : (float)bh;
    const float hx = fmaxf(lw, 1.f) * 0.5f, hy = fmaxf(lh, 1.f) * 0.5f;
    const float spx = fmaxf(lw - 1.f, 1.f) / (float)(g - 1), spy = fmaxf(lh - 1.f, 1.f) / (float)(g - 1);
    float acc[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) acc[k] = 0.f;
    for (TileWalk pw(bw, bh, gridDim.x); pw.ok(); pw.next()) {
        if (!pw.in()) continue;
        const int y = pw.y(), x = pw.x();
        const size_t t = (size_t)y * bw + x;
        float fx, fy, X, Y;
        float3 ph;
        if (!sample_pos<true>(Hi, fv, x, y, aw, ah, bw, bh, fx, fy, ph, X, Y)) continue;
        float wt, tpx, tpy;
        taper(fx, fy, (float)aw, (float)ah, wt, tpx, tpy);
        const float flx = floorf(fx), fly = floorf(fy);
        const float ax = fx - flx, ay = fy - fly;
        const size_t i00 = (size_t)(int)fly * aw + (int)flx;  // fx, fy ≥ 2 here
        float va[4], gx[4], gy[4], vb[4];
        const Taps4 tp = taps4(fa, i00, aw);
        const float4 b4 = __ldg(&fb[t]);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const float v00 = comp4(tp.v00, p), v10 = comp4(tp.v10, p);
            const float v01 = comp4(tp.v01, p), v11 = comp4(tp.v11, p);
            va[p] = (v00 * (1.f - ax) + v10 * ax) * (1.f - ay) + (v01 * (1.f - ax) + v11 * ax) * ay;
            gx[p] = (v10 - v00) * (1.f - ay) + (v11 - v01) * ay;
            gy[p] = (v01 - v00) * (1.f - ax) + (v11 - v10) * ax;
            vb[p] = comp4(b4, p);
        }
        float dga = 0.f, dgb = 0.f;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            float s = 0.f;
#pragma unroll
            for (int b = 0; b < 4; ++b) s += cf[a * 4 + b] * (vb[b] - cf[16 + b]) - cf[20 + a * 4 + b] * (va[b] - cf[36 + b]);
            dga += 2.f * s * gx[a];
            dgb += 2.f * s * gy[a];
        }
        float bwv = 0.f;
        if (tpx != 0.f || tpy != 0.f) {
            const float* gg = cf + kG0;
            float s = gg[0];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s += gg[1 + i] * va[i] + gg[5 + i] * vb[i];
#pragma unroll
                for (int j = 0; j < 4; ++j) s += gg[9 + i * 4 + j] * va[i] * vb[j];
#pragma unroll
                for (int j = i; j < 4; ++j) s += gg[25 + tri4(i, j)] * va[i] * va[j] + gg[35 + tri4(i, j)] * vb[i] * vb[j];
            }
            bwv = s;
        }
        // the sample's motion per unit basis weight of a control point's x / y displacement
        float uxx, uxy, uyx, uyy;
        float su, sv;
        if (src) {
            uxx = hx, uxy = 0.f, uyx = 0.f, uyy = hy;
            su = (ph.x / ph.z - 1.f) / spx;
            sv = (ph.y / ph.z - 1.f) / spy;
        } else {
            const float z = ph.z, z2 = fmaxf(z * z, 1e-12f);
            uxx = hx * (Hi[0] * z - ph.x * Hi[6]) / z2;
            uxy = hx * (Hi[3] * z - ph.y * Hi[6]) / z2;
            uyx = hy * (Hi[1] * z - ph.x * Hi[7]) / z2;
            uyy = hy * (Hi[4] * z - ph.y * Hi[7]) / z2;
            su = (float)x / spx;
            sv = (float)y / spy;
        }
        const float Gx = wt * (dga * uxx + dgb * uxy) + bwv * (tpx * uxx + tpy * uxy);
        const float Gy = wt * (dga * uyx + dgb * uyy) + bwv * (tpx * uyx + tpy * uyy);
        if (!(Gx == Gx) || !(Gy == Gy)) continue;
        const int iu = (int)floorf(su), iv = (int)floorf(sv);
        const float4 bu = cubic_w(fminf(fmaxf(su - (float)iu, 0.f), 1.f));
        const float4 bv = cubic_w(fminf(fmaxf(sv - (float)iv, 0.f), 1.f));
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int cp = cp0 + k;
            if (cp >= g * g) break;
            const int ci = cp % g, cj = cp / g;
            float wu = 0.f, wv = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (min(max(iu - 1 + q, 0), g - 1) == ci) wu += comp4(bu, q);
                if (min(max(iv - 1 + q, 0), g - 1) == cj) wv += comp4(bv, q);
            }
            const float bk = wu * wv;
            acc[2 * k] += bk * Gx;
            acc[2 * k + 1] += bk * Gy;
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const float v = warp_sumf(acc[k]);
        if (lane == 0) red[w][k] = v;
    }
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < 32)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += (double)red[i][threadIdx.x];
    __shared__ double tot[48];
    block_add(s, 32, out, rd, 0, gridDim.x, tot);
}

// The spline's Gauss–Newton terms of one lattice cell (smi.wgsl ffd_cells 2065-2264): block =
// (cell, chunk of its pixel tiles). The cell's fixed pixels (the cell itself on a fixed-image
// lattice; the bounding box of the moving cell's corners under H, one pixel wider, on a
// moving-image lattice) in tiles of 256: each thread stages one pixel that samples inside the
// moving image and whose lattice point lies in this cell — its basis weights, K = wt·Jdᵀ S Jd
// (S = ∇vᵀ Q ∇v, Jd the sample's motion per unit control-point displacement) and the
// gradient Jdᵀ (wt ∇S + the taper term) — then thread (task, half) adds its share of the tile:
// tasks 0–99 a pair of symmetric basis products × (K_xx, K_xy, K_yy), 100–115 a tap × ∇.
constexpr int kFcTasks = 116;
__device__ __forceinline__ int tri_i(int k) { return k < 4 ? 0 : k < 7 ? 1 : k < 9 ? 2 : 3; }
__device__ __forceinline__ int tri_j(int k) { return k < 4 ? k : k < 7 ? k - 3 : k < 9 ? k - 5 : 3; }

__global__ void __launch_bounds__(256) k_pose_ffd_cells(const float4* __restrict__ fa, int aw, int ah,
                                                        const float4* __restrict__ fb, int bw, int bh,
                                                        const float* __restrict__ hinv, const float* __restrict__ hpose,
                                                        const float* __restrict__ coef, PoseFfd ffd, int nch,
                                                        float* __restrict__ out) {
    __shared__ float Hs[9], Hp[9], cf[kCoef];
    __shared__ float cps[2 * kFfdMax * kFfdMax];
    __shared__ float4 s_bu[256], s_bv[256], s_k[256];
    __shared__ float s_gy[256];
    __shared__ float3 s_acc[256];
    if (threadIdx.x < 9) {
        Hs[threadIdx.x] = hinv[threadIdx.x];
        Hp[threadIdx.x] = hpose[threadIdx.x];
    }
    for (int k = threadIdx.x; k < kCoef; k += blockDim.x) cf[k] = coef[k];
    const FfdView fv = ffd_view(ffd, cps);
    __syncthreads();
    float Hi[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) Hi[i] = Hs[i];
    const int g = fv.g;
    const int cell = blockIdx.x / nch, chunk = blockIdx.x % nch;
    const int iu = cell % g, iv = cell / g;
    const bool src = fv.source != 0;
    const float rw = (float)bw, rh = (float)bh, sw = (float)aw, shh = (float)ah;
    const float lw = src ? sw : rw, lh = src ? shh : rh;
    const float hx = fmaxf(lw, 1.f) * 0.5f, hy = fmaxf(lh, 1.f) * 0.5f;
    const float spx = fmaxf(lw - 1.f, 1.f) / (float)(g - 1), spy = fmaxf(lh - 1.f, 1.f) / (float)(g - 1);
    float x0 = 0.f, x1 = rw - 1.f, y0 = 0.f, y1 = rh - 1.f;
    if (!src) {
        x0 = fmaxf(0.f, floorf((float)iu * spx) - 1.f);
        x1 = fminf(rw - 1.f, ceilf((float)(iu + 1) * spx) + 1.f);
        y0 = fmaxf(0.f, floorf((float)iv * spy) - 1.f);
        y1 = fminf(rh - 1.f, ceilf((float)(iv + 1) * spy) + 1.f);
    } else {
        float bx0 = 3.0e38f, bx1 = -3.0e38f, by0 = 3.0e38f, by1 = -3.0e38f;
        for (int c = 0; c < 4; ++c) {
            const float mx = (float)(iu + (c & 1)) * spx + 1.f, my = (float)(iv + (c >> 1)) * spy + 1.f;
            const float qx = Hp[0] * mx + Hp[1] * my + Hp[2], qy = Hp[3] * mx + Hp[4] * my + Hp[5];
            const float qz = Hp[6] * mx + Hp[7] * my + Hp[8];
            if (fabsf(qz) < 1e-8f) continue;
            bx0 = fminf(bx0, qx / qz - 1.f);
            bx1 = fmaxf(bx1, qx / qz - 1.f);
            by0 = fminf(by0, qy / qz - 1.f);
            by1 = fmaxf(by1, qy / qz - 1.f);
        }
        x0 = fmaxf(0.f, floorf(bx0) - 1.f);
        x1 = fminf(rw - 1.f, ceilf(bx1) + 1.f);
        y0 = fmaxf(0.f, floorf(by0) - 1.f);
        y1 = fminf(rh - 1.f, ceilf(by1) + 1.f);
    }
    const int bwx = (int)fmaxf(x1 - x0 + 1.f, 0.f), bhy = (int)fmaxf(y1 - y0 + 1.f, 0.f);
    const int total = bwx * bhy;
    const int half = threadIdx.x / kFcTasks, task = threadIdx.x % kFcTasks;
    int bi = 0, bi2 = 0, bj = 0, bj2 = 0;
    if (task < 100) {
        bi = tri_i(task / 10), bi2 = tri_j(task / 10), bj = tri_i(task % 10), bj2 = tri_j(task % 10);
    } else {
        bi = (task - 100) % 4, bj = (task - 100) / 4;
    }
    float3 acc = make_float3(0.f, 0.f, 0.f);
    const int ntile = (total + 255) / 256;
    for (int tile = chunk * ntile / nch; tile < (chunk + 1) * ntile / nch; ++tile) {
        const int base = tile * 256, pidx = base + threadIdx.x;
        bool ok = false;
        float4 bu = make_float4(0.f, 0.f, 0.f, 0.f), bv = bu, kk = bu;
        float gyv = 0.f;
        if (pidx < total) {
            const int xi = (int)x0 + pidx % bwx, yi = (int)y0 + pidx / bwx;
            float fx, fy, X, Y, su, sv;
            float3 ph;
            ok = sample_pos<true>(Hi, fv, xi, yi, aw, ah, bw, bh, fx, fy, ph, X, Y);
            if (fabsf(ph.z) >= 1e-8f) {
                if (src) {
                    su = (ph.x / ph.z - 1.f) / spx;
                    sv = (ph.y / ph.z - 1.f) / spy;
                } else {
                    su = (float)xi / spx;
                    sv = (float)yi / spy;
                }
                // this cell's pixels only (each pixel belongs to exactly one cell)
                if ((int)floorf(su) != iu || (int)floorf(sv) != iv) ok = false;
                if (su < 0.f || sv < 0.f || su > (float)(g - 1) || sv > (float)(g - 1)) ok = false;
            } else {
                ok = false;
                su = sv = 0.f;
            }
            if (ok) {
                const size_t t = (size_t)yi * bw + xi;
                float wt, tpx, tpy;
                taper(fx, fy, sw, shh, wt, tpx, tpy);
                const float flx = floorf(fx), fly = floorf(fy);
                const float ax = fx - flx, ay = fy - fly;
                const size_t i00 = (size_t)(int)fly * aw + (int)flx;  // fx, fy ≥ 2 here
                float va[4], gx[4], gy[4], vb[4];
                const Taps4 tp = taps4(fa, i00, aw);
                const float4 b4 = __ldg(&fb[t]);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const float v00 = comp4(tp.v00, p), v10 = comp4(tp.v10, p);
                    const float v01 = comp4(tp.v01, p), v11 = comp4(tp.v11, p);
                    va[p] = (v00 * (1.f - ax) + v10 * ax) * (1.f - ay) + (v01 * (1.f - ax) + v11 * ax) * ay;
                    gx[p] = (v10 - v00) * (1.f - ay) + (v11 - v01) * ay;
                    gy[p] = (v01 - v00) * (1.f - ax) + (v11 - v10) * ax;
                    vb[p] = comp4(b4, p);
                }
                float rx = 0.f, ry = 0.f;
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    float s = 0.f;
#pragma unroll
                    for (int b = 0; b < 4; ++b) s += cf[a * 4 + b] * (vb[b] - cf[16 + b]) - cf[20 + a * 4 + b] * (va[b] - cf[36 + b]);
                    rx += 2.f * s * gx[a];
                    ry += 2.f * s * gy[a];
                }
                float bwb = 0.f;
                if (tpx != 0.f || tpy != 0.f) {
                    const float* gg = cf + kG0;
                    float s = gg[0];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        s += gg[1 + i] * va[i] + gg[5 + i] * vb[i];
#pragma unroll
                        for (int j = 0; j < 4; ++j) s += gg[9 + i * 4 + j] * va[i] * vb[j];
#pragma unroll
                        for (int j = i; j < 4; ++j) s += gg[25 + tri4(i, j)] * va[i] * va[j] + gg[35 + tri4(i, j)] * vb[i] * vb[j];
                    }
                    bwb = s;
                }
                float j00, j10, j01, j11;
                if (src) {
                    j00 = hx, j10 = 0.f, j01 = 0.f, j11 = hy;
                } else {
                    const float z = ph.z, z2 = fmaxf(z * z, 1e-12f);
                    j00 = hx * (Hi[0] * z - ph.x * Hi[6]) / z2;
                    j10 = hx * (Hi[3] * z - ph.y * Hi[6]) / z2;
                    j01 = hy * (Hi[1] * z - ph.x * Hi[7]) / z2;
                    j11 = hy * (Hi[4] * z - ph.y * Hi[7]) / z2;
                }
                float sxx = 0.f, sxy = 0.f, syy = 0.f;
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    float qx = 0.f, qy = 0.f;
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        qx += cf[kQ0 + a * 4 + b] * gx[b];
                        qy += cf[kQ0 + a * 4 + b] * gy[b];
                    }
                    sxx += gx[a] * qx;
                    sxy += gx[a] * qy;
                    syy += gy[a] * qy;
                }
                const float px = wt * rx + bwb * tpx, py = wt * ry + bwb * tpy;
                const float gxv = j00 * px + j10 * py;
                gyv = j01 * px + j11 * py;
                const float a0 = sxx * j00 + sxy * j10, a1 = sxy * j00 + syy * j10;
                const float b0 = sxx * j01 + sxy * j11, b1 = sxy * j01 + syy * j11;
                kk = make_float4(wt * (j00 * a0 + j10 * a1), wt * (j00 * b0 + j10 * b1), wt * (j01 * b0 + j11 * b1), gxv);
                bu = cubic_w(fminf(fmaxf(su - floorf(su), 0.f), 1.f));
                bv = cubic_w(fminf(fmaxf(sv - floorf(sv), 0.f), 1.f));
                if (!(fabsf(kk.x) + fabsf(kk.y) + fabsf(kk.z) + fabsf(kk.w) + fabsf(gyv) < 1e30f)) ok = false;
            }
        }
        if (!ok) {
            bu = bv = kk = make_float4(0.f, 0.f, 0.f, 0.f);
            gyv = 0.f;
        }
        s_bu[threadIdx.x] = bu;
        s_bv[threadIdx.x] = bv;
        s_k[threadIdx.x] = kk;
        s_gy[threadIdx.x] = gyv;
        __syncthreads();
        const int m = min(256, total - base);
        if (half < 2) {
            const int e1 = min(m, (half + 1) * 128);
            if (task < 100) {
                for (int e = half * 128; e < e1; ++e) {
                    const float pr = comp4(s_bu[e], bi) * comp4(s_bu[e], bi2) * comp4(s_bv[e], bj) * comp4(s_bv[e], bj2);
                    acc.x += pr * s_k[e].x;
                    acc.y += pr * s_k[e].y;
                    acc.z += pr * s_k[e].z;
                }
            } else {
                for (int e = half * 128; e < e1; ++e) {
                    const float b = comp4(s_bu[e], bi) * comp4(s_bv[e], bj);
                    acc.x += s_k[e].w * b;
                    acc.y += s_gy[e] * b;
                }
            }
        }
        __syncthreads();
    }
    s_acc[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x < kFcTasks) {
        const float3 u = s_acc[threadIdx.x], v = s_acc[threadIdx.x + kFcTasks];
        float* o = out + (size_t)blockIdx.x * kFfdCell;
        if (threadIdx.x < 100) {
            o[threadIdx.x * 3] = u.x + v.x;
            o[threadIdx.x * 3 + 1] = u.y + v.y;
            o[threadIdx.x * 3 + 2] = u.z + v.z;
        } else {
            o[300 + (threadIdx.x - 100) * 2] = u.x + v.x;
            o[300 + (threadIdx.x - 100) * 2 + 1] = u.y + v.y;
        }
    }
}

// Blocks per pose over `pixels` fixed pixels, with `slots` blocks resident on the GPU at once:
// about 16 pixels per thread, rounded so that whole poses fill whole waves (slots / b poses per
// wave, or b a whole number of waves) — a wave and a few blocks would take two waves' time. The
// count depends on the image alone, never on how many poses share the launch, so a pose's sums
// (and score) are the same whatever batch it is scored in.
// zc_tune_parts' knobs (0 keeps the default): pixels per thread (16), the least and the most
// blocks per pose (none, 4096)
std::atomic<unsigned> g_px_per_thread{16}, g_min_blocks{0}, g_max_blocks{4096};

int pose_blocks(size_t pixels, int slots) {
    const size_t ppt = std::max(1u, g_px_per_thread.load(std::memory_order_relaxed));
    const size_t by_work = std::max<size_t>(1, (pixels + 256 * ppt - 1) / (256 * ppt));
    const size_t sl = (size_t)std::max(slots, 1);
    size_t b = by_work >= sl ? sl * (by_work / sl) : sl / ((sl + by_work - 1) / by_work);
    b = std::max<size_t>(b, g_min_blocks.load(std::memory_order_relaxed));
    return (int)std::max<size_t>(1, std::min<size_t>(b, std::max(1u, g_max_blocks.load(std::memory_order_relaxed))));
}

// resident blocks of 256 threads of kernel k across the GPU
template <class K>
int pose_slots(K k) {
    int dev = 0, sms = 148, per = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, 256, 0) != cudaSuccess || per < 1) per = 1;
    return per * sms;
}

}  // namespace

void pose_tune(unsigned px_per_thread, unsigned min_blocks, unsigned max_blocks) {
    if (px_per_thread) g_px_per_thread = std::min(px_per_thread, 4096u);
    if (min_blocks) g_min_blocks = std::min(min_blocks, 4096u);
    if (max_blocks) g_max_blocks = std::min(max_blocks, 4096u);
}

namespace {
// resident blocks of each pose kernel: moments (spline, plain), tangent (spline, plain), ffd_grad
const std::array<int, 5>& kernel_slots() {
    static const std::array<int, 5> sl{pose_slots(k_pose_moments<true, 1>), pose_slots(k_pose_moments<false, 1>),
                                       pose_slots(k_pose_tangent<true>), pose_slots(k_pose_tangent<false>),
                                       pose_slots(k_pose_ffd_grad)};
    return sl;
}
// part must hold n poses × blocks × k totals and ticket n counters
bool red_fits(const PoseRed& r, int n, int blocks, int k) {
    return !r.part || (r.ticket && r.tickets >= (size_t)n && r.cap >= (size_t)n * blocks * k);
}
}  // namespace

size_t pose_red_need(size_t pixels, int n) {
    int b = 1;
    for (int sl : kernel_slots()) b = std::max(b, pose_blocks(pixels, sl));
    return (size_t)std::max(n, 1) * b * kMom;
}

namespace {
// the call's images, blocks per row and poses; g.y: the poses of a launch, as many as the scratch holds
// rows for (and a grid has rows). A pose's sums do not depend on which poses share its launch.
cudaError_t pose_launch(const PoseCall& c, int slot, int k, PoseLaunch& L, dim3& g) {
    for (const PoseFfd& f : c.ffd)
        if (f.cps && (f.g < 2 || f.g > kFfdMax)) return cudaErrorInvalidValue;
    const int nd = c.sym ? 2 : 1;
    const PoseSide* side[2] = {&c.a, &c.b};
    g = dim3(1, 1, nd);
    for (int d = 0; d < 2; ++d) {
        L.f[d] = side[d]->feat4, L.w[d] = side[d]->w, L.h[d] = side[d]->h;
        const PoseSide& dst = *side[1 - d];
        L.nblk[d] = pose_blocks((size_t)dst.w * dst.h, kernel_slots()[slot]);
        if (d < nd) g.x = std::max(g.x, (unsigned)L.nblk[d]);
        L.ffd[d] = c.ffd[d];
    }
    if (!red_fits(c.red, nd, (int)g.x, k)) return cudaErrorInvalidValue;
    g.y = (unsigned)std::min(c.n, 65535);
    if (c.red.part) g.y = (unsigned)std::min<size_t>(g.y, std::min(c.red.tickets, c.red.cap / ((size_t)g.x * k)) / nd);
    L.n = c.n, L.hinv = c.hinv, L.mask = c.mask, L.rd = c.red;
    L.n_inl = c.hinv_host && nd * c.n <= kPoseInline ? nd * c.n : 0;
    for (int i = 0; i < 9 * L.n_inl; ++i) L.inl[i] = c.hinv_host[i];
    return cudaSuccess;
}

// launch(grid, poses) for every g.y poses of the call, in order
template <class K>
cudaError_t pose_launches(int n, dim3 g, PoseLaunch& L, K&& launch) {
    for (const int step = (int)g.y; L.p0 < n; L.p0 += step) {
        g.y = (unsigned)std::min(step, n - L.p0);
        launch(g);
        if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
}  // namespace

cudaError_t pose_moments(const PoseCall& c, double* sums, const PoseScores& sc, cudaStream_t st) {
    if (c.n <= 0) return cudaSuccess;
    const bool ffd = c.ffd[0].cps || c.ffd[1].cps;
    PoseLaunch L{};
    dim3 g;
    cudaError_t e = pose_launch(c, ffd ? 0 : 1, kMom, L, g);
    if (e != cudaSuccess) return e;
    L.out = sums, L.host = sc.host_sums;
    L.scored = sc.score != nullptr && c.red.part, L.exact = sc.exact ? 1 : 0;
    L.coef = sc.coef, L.score = sc.score, L.host_score = sc.host_score;
    if (!c.red.part && (e = cudaMemsetAsync(sums, 0, (size_t)c.n * g.z * kMom * sizeof(double), st)) != cudaSuccess) return e;
    // Launches of fewer blocks than SMs (a pose or two of an ordinary image) keep four pixels' taps in
    // flight: a 256² pair's score takes 33 µs from call to result, 36 with one. Fuller launches lose
    // more warps to the registers than they gain (two pixels: 8 % slower).
    return pose_launches(c.n, g, L, [&](dim3 b) {
        if (ffd) k_pose_moments<true, 1><<<b, 256, 0, st>>>(L);
        else if ((int)(b.x * b.y * b.z) <= kernel_slots()[1] / 3) k_pose_moments<false, 4><<<b, 256, 0, st>>>(L);
        else k_pose_moments<false, 1><<<b, 256, 0, st>>>(L);
    });
}

cudaError_t pose_tangent(const PoseCall& c, const float* coef, const float* gens, bool hess, double* out, double* host,
                         cudaStream_t st) {
    if (c.n <= 0) return cudaSuccess;
    const bool ffd = c.ffd[0].cps || c.ffd[1].cps;
    PoseLaunch L{};
    dim3 g;
    cudaError_t e = pose_launch(c, ffd ? 2 : 3, kGrad, L, g);
    if (e != cudaSuccess) return e;
    L.out = out, L.host = host, L.coef = const_cast<float*>(coef), L.hess = hess ? 1 : 0;
    for (int i = 0; i < 144; ++i) L.gens[i] = gens[i];
    if (!c.red.part && (e = cudaMemsetAsync(out, 0, (size_t)c.n * g.z * kGrad * sizeof(double), st)) != cudaSuccess) return e;
    return pose_launches(c.n, g, L, [&](dim3 b) {
        if (ffd) k_pose_tangent<true><<<b, 256, 0, st>>>(L);
        else k_pose_tangent<false><<<b, 256, 0, st>>>(L);
    });
}

cudaError_t pose_ffd_cells(const PoseSide& a, const PoseSide& b, const float* hinv, const float* hpose,
                           const float* coef, const PoseFfd& ffd, int nch, float* out, cudaStream_t st) {
    if (!ffd.cps || ffd.g < 2 || ffd.g > kFfdMax || nch < 1) return cudaErrorInvalidValue;
    k_pose_ffd_cells<<<ffd.g * ffd.g * nch, 256, 0, st>>>(a.feat4, a.w, a.h, b.feat4, b.w, b.h, hinv, hpose, coef, ffd,
                                                          nch, out);
    return cudaGetLastError();
}

cudaError_t pose_ffd_grad(const PoseSide& a, const PoseSide& b, const float* hinv, const float* coef,
                          const PoseFfd& ffd, int cp0, double* out, cudaStream_t st, const PoseRed& red) {
    if (!ffd.cps || ffd.g < 2 || ffd.g > kFfdMax) return cudaErrorInvalidValue;
    const int blocks = pose_blocks((size_t)b.w * b.h, kernel_slots()[4]);
    if (!red_fits(red, 1, blocks, 32)) return cudaErrorInvalidValue;
    cudaMemsetAsync(out, 0, 32 * sizeof(double), st);
    k_pose_ffd_grad<<<blocks, 256, 0, st>>>(a.feat4, a.w, a.h, b.feat4, b.w, b.h, hinv, coef, ffd, cp0, out, red);
    return cudaGetLastError();
}

cudaError_t pose_coefs(const double* sums, int n, bool exact, float* coef, double* score, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_pose_coefs<<<(n + 3) / 4, 128, 0, st>>>(sums, n, exact ? 1 : 0, 1e-4, coef, score);
    return cudaGetLastError();
}

}  // namespace zc
