// Line FFTs in shared memory for the SMI maps.
//
// A line of n complex points (n = 2^a·3^b, the reference's "ladder" sizes, src/fft.zig:14-34)
// is transformed in place in shared memory by a Stockham autosort schedule of radix-16/8/4/2/3
// stages (radices 16, 8, 4, 2 for the power of two, 3 for each factor 3). Each stage reads every
// butterfly's inputs into registers, synchronises, then twiddles, runs the small DFT and writes
// the outputs at their autosorted places, so one buffer of n points serves all stages.
// Forward: e^{−2πi k t/n}, no scaling; inverse: e^{+2πi k t/n}, no scaling (the 1/(nx·ny) of
// src/fft.zig:280-286 is applied where the correlations are scored).
//
// Shared-memory index padding (one slot per 16 points) keeps the strided writes of the first
// stages free of bank conflicts.
#pragma once

#include "common.cuh"

namespace zc {

constexpr int kMaxStages = 16;
constexpr int kMaxLine = 8192;

struct LinePlan {
    int n;                    // line length
    int nst;                  // number of stages
    int radix[kMaxStages];    // radix of each stage, in order
    int tl;                   // threads per line (each stage's butterflies fit in tl·16/R)
    const float2* tw;         // n twiddles e^{−2πi t/n}, t < n (device memory)
    int s0 = 0;               // first stage run: stages before it were applied by another pass
};

__host__ __device__ __forceinline__ constexpr int pad_idx(int i) { return i + (i >> 4); }
__host__ __device__ __forceinline__ constexpr int padded_len(int n) { return n + (n >> 4) + 1; }
// pitch between lines stored side by side (column tiles): ≡ 4 (mod 16) points, so a half-warp
// touching 4 lines × 4 consecutive points hits 16 distinct bank pairs
__host__ __device__ __forceinline__ constexpr int line_pitch(int n) {
    const int p = padded_len(n);
    return p + ((4 - (p & 15)) & 15);
}

// Pitch between the tx lines of a column tile whose threads run column-fastest (line c = thread
// mod tx): a half-warp then touches min(tx, 16) lines at 16 / min(tx, 16) consecutive points each,
// and the pitch puts them in distinct bank pairs — ≡ 16/tx (mod 16) for tx = 2, 4, 8, odd for
// 16 or more lines (or a count that is not a power of two), where each line is touched once.
__host__ __device__ __forceinline__ constexpr int tile_pitch(int n, int tx) {
    return (tx >= 16 || (tx & (tx - 1)) != 0) ? (padded_len(n) | 1)
                                               : padded_len(n) + (((16 / tx) - (padded_len(n) & 15)) & 15);
}

// Padded slots of the points i0 + r·D (r = 0, 1, ...) from p0 = pad_idx(i0), for a compile-time
// step D, folded to constant offsets: when D is a multiple of 16 every step adds D + D/16; when
// all the points lie in one aligned group of 16 (the caller guarantees it) every step adds D.
template <int D, bool ONE_GROUP = false>
__device__ __forceinline__ int pad_at(int p0, int r) {
    static_assert(D % 16 == 0 || ONE_GROUP, "steps that cross 16-point groups need pad_idx");
    return p0 + r * (D % 16 == 0 ? D + D / 16 : D);
}

// The padded slot of output r of first-stage butterfly j (point j·R0 + r): one aligned group of
// 16 holds the butterfly when R0 divides 16.
template <int R0>
__device__ __forceinline__ int first_slot(int j, int r) {
    if constexpr (16 % R0 == 0) return pad_at<1, true>(pad_idx(j * R0), r);
    else return pad_idx(j * R0 + r);
}

// ── small DFTs, natural order in and out; INV flips the sign of the exponent ──

template <bool INV>
__device__ __forceinline__ float2 mul_mi(float2 a) {  // a·(−i) forward, a·(+i) inverse
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft2(float2* v) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
}

template <bool INV>
__device__ __forceinline__ void dft3(float2* v) {
    const float s3 = 0.86602540378443864676f;
    const float2 t = cadd(v[1], v[2]);
    const float2 d = csub(v[1], v[2]);
    const float2 m = make_float2(v[0].x - 0.5f * t.x, v[0].y - 0.5f * t.y);
    const float2 j = mul_mi<INV>(cscale(d, s3));
    v[0] = cadd(v[0], t);
    v[1] = cadd(m, j);
    v[2] = csub(m, j);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2* v) {
    const float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
    const float2 a2 = cadd(v[1], v[3]), a3 = mul_mi<INV>(csub(v[1], v[3]));
    v[0] = cadd(a0, a2);
    v[2] = csub(a0, a2);
    v[1] = cadd(a1, a3);
    v[3] = csub(a1, a3);
}

// dft8 after its first butterfly layer: a_r = v_r + v_{r+4}, b_r = v_r − v_{r+4}
template <bool INV>
__device__ __forceinline__ void dft8_ab(float2 (&a)[4], float2 (&b)[4], float2* v) {
    const float h = 0.70710678118654752440f;
    // b_r ·= w8^r
    b[1] = INV ? make_float2(h * (b[1].x - b[1].y), h * (b[1].x + b[1].y))
               : make_float2(h * (b[1].x + b[1].y), h * (b[1].y - b[1].x));
    b[2] = mul_mi<INV>(b[2]);
    b[3] = INV ? make_float2(-h * (b[3].x + b[3].y), h * (b[3].x - b[3].y))
               : make_float2(h * (b[3].y - b[3].x), -h * (b[3].x + b[3].y));
    dft4<INV>(a);
    dft4<INV>(b);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[2 * k] = a[k];
        v[2 * k + 1] = b[k];
    }
}

template <bool INV>
__device__ __forceinline__ void dft8(float2* v) {
    float2 a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        a[r] = cadd(v[r], v[r + 4]);
        b[r] = csub(v[r], v[r + 4]);
    }
    dft8_ab<INV>(a, b, v);
}

// dft16 after its first butterfly layer: a_r = v_r + v_{r+8}, d_r = v_r − v_{r+8}
template <bool INV>
__device__ __forceinline__ void dft16_ad(float2 (&a)[8], float2 (&d)[8], float2* v) {
    // w16^r = (cos 2πr/16, ∓sin 2πr/16), r = 0..7
    const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
    const float h = 0.70710678118654752440f;
    const float cs[8] = {1.f, c1, h, s1, 0.f, -s1, -h, -c1};
    const float sn[8] = {0.f, s1, h, c1, 1.f, c1, h, s1};
    float2 b[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const float si = INV ? sn[r] : -sn[r];
        b[r] = make_float2(d[r].x * cs[r] - d[r].y * si, d[r].x * si + d[r].y * cs[r]);
    }
    dft8<INV>(a);
    dft8<INV>(b);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        v[2 * k] = a[k];
        v[2 * k + 1] = b[k];
    }
}

template <bool INV>
__device__ __forceinline__ void dft16(float2* v) {
    float2 a[8], d[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        a[r] = cadd(v[r], v[r + 8]);
        d[r] = csub(v[r], v[r + 8]);
    }
    dft16_ad<INV>(a, d, v);
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2* v) {
    if constexpr (R == 2) dft2<INV>(v);
    else if constexpr (R == 3) dft3<INV>(v);
    else if constexpr (R == 4) dft4<INV>(v);
    else if constexpr (R == 8) dft8<INV>(v);
    else dft16<INV>(v);
}

// The small DFT of R points whose upper half (v_r, r ≥ R/2) is zero and is not read: the first
// butterfly layer reduces to copies (zero-padded lines: their first stage reads half the points).
template <int R, bool INV>
__device__ __forceinline__ void dft_lo(float2* v) {
    static_assert(R % 2 == 0, "an odd radix has no zero half");
    if constexpr (R == 16) {
        float2 a[8], d[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) a[r] = d[r] = v[r];
        dft16_ad<INV>(a, d, v);
    } else if constexpr (R == 8) {
        float2 a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) a[r] = b[r] = v[r];
        dft8_ab<INV>(a, b, v);
    } else if constexpr (R == 4) {
        const float2 a = v[0], b = v[1], mb = mul_mi<INV>(v[1]);
        v[0] = cadd(a, b);
        v[1] = cadd(a, mb);
        v[2] = csub(a, b);
        v[3] = csub(a, mb);
    } else {
        v[1] = v[0];
    }
}

// One Stockham stage of radix R over a line in shared memory. Thread `t` of the line's `tlc`
// threads takes butterflies j = t + b·tlc, b < BM (BM·R ≤ 18 registers of points). Ns: the
// length of the sub-transforms done so far. All threads of the block must call it (it holds two
// __syncthreads); threads without a line pass t ≥ 2^30.
template <int R, int BM, bool INV>
__device__ __noinline__ void fft_stage(float2* __restrict__ buf, const float2* __restrict__ tw,
                                          int n, int Ns, int t, int tlc) {
    const int m = n / R;
    const int tws = n / (Ns * R);
    float2 v[BM][R];
#pragma unroll
    for (int b = 0; b < BM; ++b) {
        const int j = t + b * tlc;
        if (j < m) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[b][r] = buf[pad_idx(j + r * m)];
        }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < BM; ++b) {
        const int j = t + b * tlc;
        if (j < m) {
            const int k = j % Ns;
            if (Ns > 1) {
#pragma unroll
                for (int r = 1; r < R; ++r) {
                    float2 w = __ldg(&tw[r * k * tws]);
                    if (INV) w.y = -w.y;
                    v[b][r] = cmul(v[b][r], w);
                }
            }
            dft<R, INV>(v[b]);
            const int base = (j - k) * R + k;
#pragma unroll
            for (int r = 0; r < R; ++r) buf[pad_idx(base + r * Ns)] = v[b][r];
        }
    }
    __syncthreads();
}

// The whole line: every thread of the block calls it; `t` is the thread's index within its
// line's plan.tl threads (≥ 2^30 for threads without a line).
template <bool INV>
__device__ __forceinline__ void line_fft(float2* __restrict__ buf, const LinePlan& p, int t) {
    int Ns = 1;
    for (int s = 0; s < p.s0; ++s) Ns *= p.radix[s];
    for (int s = p.s0; s < p.nst; ++s) {
        const int R = p.radix[s];
        switch (R) {
            case 16: fft_stage<16, 1, INV>(buf, p.tw, p.n, Ns, t, p.tl); break;
            case 8: fft_stage<8, 2, INV>(buf, p.tw, p.n, Ns, t, p.tl); break;
            case 4: fft_stage<4, 4, INV>(buf, p.tw, p.n, Ns, t, p.tl); break;
            case 2: fft_stage<2, 8, INV>(buf, p.tw, p.n, Ns, t, p.tl); break;
            default: fft_stage<3, 6, INV>(buf, p.tw, p.n, Ns, t, p.tl); break;
        }
        Ns *= R;
    }
}

// ── lines of N = 2^a·3^b points with the whole schedule known at compile time ──
// ⌈a/4⌉ power-of-two stages with balanced radices (16/8/4/2), then b radix-3 stages; TL threads
// per line, each taking ⌈(N/R)/TL⌉ butterflies of a radix-R stage. Strides, twiddle steps and
// index arithmetic fold to constants.
constexpr int ilog2(int n) { return n <= 1 ? 0 : 1 + ilog2(n >> 1); }
constexpr int twos_of(int n) { return (n > 0 && n % 2 == 0) ? 1 + twos_of(n / 2) : 0; }
constexpr int threes_of(int n) { return (n > 0 && n % 3 == 0) ? 1 + threes_of(n / 3) : 0; }
constexpr int ipow(int b, int e) { return e == 0 ? 1 : b * ipow(b, e - 1); }

// The schedule of a line of n = 2^a·3^b points (compile-time for the kernels, run-time for the
// host building the twiddle tables): the number of stages and stage s's radix.
__host__ __device__ constexpr int mix_stages(int n) { return (twos_of(n) + 3) / 4 + threes_of(n); }
__host__ __device__ constexpr int mix_radix(int n, int s) {
    return s < (twos_of(n) + 3) / 4
               ? 1 << (twos_of(n) / ((twos_of(n) + 3) / 4) + (s < twos_of(n) % ((twos_of(n) + 3) / 4) ? 1 : 0))
               : 3;
}
// Per-stage twiddle tables, after the n entries e^{−2πi t/n} of a line's table: stage s (radix R,
// NS points transformed before it, NS > 1) holds w(r, k) = e^{−2πi r k/(NS·R)} at
// (r − 1)·NS + k, r = 1..R−1, k < NS, so the threads of a stage (consecutive k) read consecutive
// entries. stage_tw_off: where stage s's table starts (past the n entries); its value at
// s = mix_stages(n) is the tables' total length.
__host__ __device__ constexpr int stage_tw_off(int n, int s) {
    int off = 0, ns = 1;
    for (int i = 0; i < s; ++i) {
        const int r = mix_radix(n, i);
        if (ns > 1) off += (r - 1) * ns;
        ns *= r;
    }
    return off;
}

template <int N>
struct Mix {
    static constexpr int kA = twos_of(N), kB = threes_of(N);
    static_assert(ipow(2, twos_of(N)) * ipow(3, threes_of(N)) == N, "line length must be 2^a·3^b");
    static constexpr int kP2 = (kA + 3) / 4;
    static constexpr int kStages = kP2 + kB;
    static_assert(kStages == mix_stages(N), "stage count");
    static constexpr int radix(int s) { return mix_radix(N, s); }
};

// Several consecutive stages run in registers as one pass through shared memory: the stages
// S .. S + CNT − 1 of radices R_S, …, product P, take the P points j + t·N/P of group j and leave
// the P outputs of the last of them, NS apart (the same butterflies, twiddles and rounding as
// stage by stage, with CNT − 1 fewer exchanges and barriers). Lines with factors of 3 need it:
// 1458 = 2·3⁶ is 7 stages but 3 passes (18 · 9 · 9). P ≤ 18 keeps a thread's points and twiddles
// within the 64 registers that two 512-thread blocks per SM leave. A 1296 × 1536 map's passes
// against the runtime plan: inverse columns 801 → 386 µs, forward rows 584 → 121, forward columns
// 538 → 152.
constexpr int kGroupMax = 18;
__host__ __device__ constexpr int radix_prod(int n, int s, int cnt) {
    int p = 1;
    for (int i = 0; i < cnt; ++i) p *= mix_radix(n, s + i);
    return p;
}
// the split of stages s.. into groups: the fewest groups, then the most even products
__host__ __device__ constexpr int group_cost(int n, int s) {
    if (s >= mix_stages(n)) return 0;
    int best = 1 << 30;
    for (int c = 1; s + c <= mix_stages(n); ++c) {
        const int p = radix_prod(n, s, c);
        if (c > 1 && p > kGroupMax) break;
        const int v = 100000 + p * p + group_cost(n, s + c);
        if (v < best) best = v;
    }
    return best;
}
__host__ __device__ constexpr int group_len(int n, int s) {
    for (int c = 1; s + c <= mix_stages(n); ++c) {
        const int p = radix_prod(n, s, c);
        if (c > 1 && p > kGroupMax) break;
        if (100000 + p * p + group_cost(n, s + c) == group_cost(n, s)) return c;
    }
    return 1;
}
// Threads per line: as many as leave every thread at most 18 points of each pass (N/16 for a power
// of two), and no more than a block's 512.
__host__ __device__ constexpr int line_tl(int n) {
    int tl = 1;
    for (int s = 0; s < mix_stages(n); s += group_len(n, s)) {
        const int p = radix_prod(n, s, group_len(n, s)), per = kGroupMax / p, t = (n / p + per - 1) / per;
        if (t > tl) tl = t;
    }
    return tl < 512 ? tl : 512;
}

// Threads per line of the inverse columns: one group of a pass each where no group has more than 9
// points (192 = 8·8·3, 576 = 8·8·9) and a line's block stays small, so that 40 registers hold a thread
// and twice the loads are in flight; else as line_tl. Inverse columns of 192²: 409 → 351 µs, of 576²
// 27 → 23; of 729² (81 threads) they lost 3 %, of 1536² (192) a third.
__host__ __device__ constexpr int col_inv_tl(int n) {
    int most = 0;
    for (int s = 0; s < mix_stages(n); s += group_len(n, s)) {
        const int p = radix_prod(n, s, group_len(n, s));
        if (p > 9) return line_tl(n);
        if (p > 3 && n / p > most) most = n / p;
    }
    return most > 0 && most <= 72 ? most : line_tl(n);
}

// Threads per line of the inverse rows: short lines' rounded up to a power of two where that adds a third
// at most, so that no line lies across two warps, whose loads and stores of a row are then whole
// aligned pieces (192 points, 12 → 16 threads: 410 → 365 µs for 104 sweep maps; 144, 9 → 16: 5 % slower).
__host__ __device__ constexpr int row_tl(int n) {
    const int tl = line_tl(n);
    int p = 1;
    while (p < tl) p *= 2;
    return tl < 32 && 3 * p <= 4 * tl ? p : tl;
}

// Stages S .. S + CNT − 1 on the P points v of group k (k = j mod NS), in registers. LO: the
// points v[t], t ≥ P/2, are zero (the line's upper half; only for an even first radix).
template <int N, int S, int CNT, int NS, bool INV, bool LO, int P>
__device__ __forceinline__ void group_apply(float2 (&v)[P], const float2* __restrict__ tw, int k) {
    static_assert(P == radix_prod(N, S, CNT), "points of the group");
    if constexpr (CNT == 1) {
        if constexpr (NS > 1) {
#pragma unroll
            for (int r = 1; r < P; ++r) {
                float2 w = __ldg(&tw[N + stage_tw_off(N, S) + (r - 1) * NS + k]);
                if (INV) w.y = -w.y;
                v[r] = cmul(v[r], w);
            }
        }
        if constexpr (LO && P % 2 == 0) dft_lo<P, INV>(v);
        else dft<P, INV>(v);
    } else {
        constexpr int RL = mix_radix(N, S + CNT - 1), PP = P / RL, NSL = NS * PP;
        float2 y[RL][PP];
#pragma unroll
        for (int l = 0; l < RL; ++l) {
            float2 q[PP];
#pragma unroll
            for (int p = 0; p < PP; ++p) q[p] = v[l + RL * p];
            group_apply<N, S, CNT - 1, NS, INV, LO, PP>(q, tw, k);
#pragma unroll
            for (int p = 0; p < PP; ++p) y[l][p] = q[p];
        }
#pragma unroll
        for (int u = 0; u < PP; ++u) {
            float2 z[RL];
            z[0] = y[0][u];
#pragma unroll
            for (int l = 1; l < RL; ++l) {
                z[l] = y[l][u];
                if (NS > 1 || u > 0) {  // else the twiddle is 1
                    float2 w = __ldg(&tw[N + stage_tw_off(N, S + CNT - 1) + (l - 1) * NSL + k + NS * u]);
                    if (INV) w.y = -w.y;
                    z[l] = cmul(z[l], w);
                }
            }
            dft<RL, INV>(z);
#pragma unroll
            for (int l = 0; l < RL; ++l) v[u + PP * l] = z[l];
        }
    }
}

// The P points of group j, N/P apart, from the line buffer.
template <int P, int N>
__device__ __forceinline__ void group_load(float2 (&v)[P], const float2* __restrict__ buf, int j) {
    constexpr int M = N / P;
    if constexpr (M % 16 == 0) {
        const int p = pad_idx(j);
#pragma unroll
        for (int r = 0; r < P; ++r) v[r] = buf[pad_at<M>(p, r)];
    } else {
#pragma unroll
        for (int r = 0; r < P; ++r) v[r] = buf[pad_idx(j + r * M)];
    }
}
// The P outputs of group j to the line buffer, NS apart from (j − k)·P + k.
template <int P, int NS>
__device__ __forceinline__ void group_store(const float2 (&v)[P], float2* __restrict__ buf, int j, int k) {
    const int base = (j - k) * P + k;
    // outputs NS apart; when P·NS divides 16 they lie in one aligned group of 16 (k < NS)
    if constexpr (NS % 16 == 0 || 16 % (P * NS) == 0) {
        const int p = pad_idx(base);
#pragma unroll
        for (int r = 0; r < P; ++r) buf[pad_at<NS, (NS % 16 != 0)>(p, r)] = v[r];
    } else {
#pragma unroll
        for (int r = 0; r < P; ++r) buf[pad_idx(base + r * NS)] = v[r];
    }
}

// One pass of a compile-time line through its buffer: the stages from S that share it.
template <int N, int TL, bool INV, int S, int NS>
__device__ __forceinline__ void mix_stage(float2* __restrict__ buf, const float2* __restrict__ tw, int t, bool act) {
    constexpr int CNT = group_len(N, S), P = radix_prod(N, S, CNT), M = N / P, BM = (M + TL - 1) / TL;
    float2 v[BM][P];
    if (act) {
#pragma unroll
        for (int b = 0; b < BM; ++b) {
            const int j = t + b * TL;
            if (M % TL == 0 || j < M) group_load<P, N>(v[b], buf, j);
        }
    }
    __syncthreads();
    if (act) {
#pragma unroll
        for (int b = 0; b < BM; ++b) {
            const int j = t + b * TL;
            if (M % TL == 0 || j < M) {
                const int k = j % NS;
                group_apply<N, S, CNT, NS, INV, false, P>(v[b], tw, k);
                group_store<P, NS>(v[b], buf, j, k);
            }
        }
    }
    __syncthreads();
}

// the passes from stage S to the end (LAST) or up to the last one
template <int N, int TL, bool INV, int S, int NS, bool LAST>
__device__ __forceinline__ void mix_run(float2* __restrict__ buf, const float2* __restrict__ tw, int t, bool act) {
    if constexpr (S < Mix<N>::kStages && (LAST || S + group_len(N, S) < Mix<N>::kStages)) {
        constexpr int CNT = group_len(N, S), P = radix_prod(N, S, CNT);
        mix_stage<N, TL, INV, S, NS>(buf, tw, t, act);
        mix_run<N, TL, INV, S + CNT, NS * P, LAST>(buf, tw, t, act);
    }
}

// the first stage of the last group
__host__ __device__ constexpr int last_group(int n) {
    int s = 0;
    while (s + group_len(n, s) < mix_stages(n)) s += group_len(n, s);
    return s;
}

// the last pass of a compile-time line, its outputs to out(y, v)
template <int N, int TL, bool INV, class Out>
__device__ __forceinline__ void mix_last(float2* __restrict__ buf, const float2* __restrict__ tw, int t, bool act,
                                         Out&& out) {
    constexpr int S = last_group(N), CNT = group_len(N, S), P = radix_prod(N, S, CNT), M = N / P, BM = (M + TL - 1) / TL;
    if (act) {
#pragma unroll 1
        for (int b = 0; b < BM; ++b) {
            const int j = t + b * TL;
            if (M % TL == 0 || j < M) {
                float2 v[P];
                group_load<P, N>(v, buf, j);
                group_apply<N, S, CNT, M, INV, false, P>(v, tw, j);  // k = j mod M = j
#pragma unroll
                for (int r = 0; r < P; ++r) out(j + r * M, v[r]);
            }
        }
    }
}

// The first pass's groups, their points from in(y), y = j + t·N/P (with LO and an even first
// radix only the lower half is read), their outputs to the line buffer.
template <int N, int TL, bool INV, bool LO, class In>
__device__ __forceinline__ void mix_first(float2* __restrict__ buf, const float2* __restrict__ tw, int t, bool act, In& in) {
    constexpr int CNT = group_len(N, 0), P = radix_prod(N, 0, CNT), M = N / P, BM = (M + TL - 1) / TL;
    constexpr bool HALF = LO && mix_radix(N, 0) % 2 == 0;
    if (act) {
#pragma unroll
        for (int b = 0; b < BM; ++b) {
            const int j = t + b * TL;
            if (M % TL == 0 || j < M) {
                float2 v[P];
#pragma unroll
                for (int r = 0; r < P; ++r) v[r] = HALF && r >= P / 2 ? make_float2(0.f, 0.f) : in(j + r * M);
                group_apply<N, 0, CNT, 1, INV, HALF, P>(v, tw, 0);
                group_store<P, 1>(v, buf, j, 0);
            }
        }
    }
}

// The whole line with its ends in registers: the first pass's groups take their inputs straight
// from in(y) (point y of the line, typically a global load) and the last pass hands its outputs
// to out(y, v), so neither end is staged through shared memory. Every thread of the block calls
// it; buf is this thread's line buffer (padded_len(N) points). On return the buffer may still be
// read by other threads of the line: synchronise before reusing it.
template <int N, int TL, bool INV, bool LO = false, class In, class Out>
__device__ __forceinline__ void mix_fft_io(float2* __restrict__ buf, const float2* __restrict__ tw, int t, bool act,
                                           In&& in, Out&& out) {
    constexpr int CNT = group_len(N, 0);
    static_assert(CNT < Mix<N>::kStages, "a line of one pass has no shared-memory exchange");
    mix_first<N, TL, INV, LO>(buf, tw, t, act, in);
    __syncthreads();
    mix_run<N, TL, INV, CNT, radix_prod(N, 0, CNT), false>(buf, tw, t, act);
    mix_last<N, TL, INV>(buf, tw, t, act, out);
}

// The whole line with its first pass fed from in(y) (as mix_fft_io) and the result left in buf
// in natural order, the block synchronised, as run() leaves it.
template <int N, int TL, bool INV, bool LO = false, class In>
__device__ __forceinline__ void mix_fft_in(float2* __restrict__ buf, const float2* __restrict__ tw, int t, bool act,
                                           In&& in) {
    constexpr int CNT = group_len(N, 0);
    mix_first<N, TL, INV, LO>(buf, tw, t, act, in);
    __syncthreads();
    mix_run<N, TL, INV, CNT, radix_prod(N, 0, CNT), true>(buf, tw, t, act);
}

// Line-FFT policies the map kernels are written against: n(), threads per line,
// run_io<INV, LO>(buf, t, act, in, out) (mix_fft_io's contract) and run_in<INV, LO>(buf, t, act,
// in); LO: the caller guarantees in(y) = 0 for y ≥ n/2, so a compile-time line reads only y < n/2.
struct GenericLine {
    static constexpr int kTl = 0, kTx = 0, kRowT = 512;  // kTx 0: tile and threads chosen at the launch
    static constexpr bool kLong = false;
    __host__ GenericLine inv() const { return *this; }
    __host__ GenericLine row() const { return *this; }
    LinePlan p;
    __device__ __forceinline__ const GenericLine& fresh() const { return *this; }
    __host__ __device__ __forceinline__ int n() const { return p.n; }
    __host__ __device__ __forceinline__ int tl() const { return p.tl; }
    // runtime lines stage through shared memory around the transform (LO: no shortcut)
    template <bool INV, bool LO = false, class In, class Out>
    __device__ __forceinline__ void run_io(float2* buf, int t, bool act, In&& in, Out&& out) const {
        const bool a = act && t < p.tl;
        if (a)
            for (int y = t; y < p.n; y += p.tl) buf[pad_idx(y)] = in(y);
        __syncthreads();
        line_fft<INV>(buf, p, a ? t : (1 << 30));
        if (a)
            for (int y = t; y < p.n; y += p.tl) out(y, buf[pad_idx(y)]);
    }
    template <bool INV, bool LO = false, class In>
    __device__ __forceinline__ void run_in(float2* buf, int t, bool act, In&& in) const {
        const bool a = act && t < p.tl;
        if (a)
            for (int y = t; y < p.n; y += p.tl) buf[pad_idx(y)] = in(y);
        __syncthreads();
        line_fft<INV>(buf, p, a ? t : (1 << 30));
    }
};

// A compile-time line of N = 2^a·3^b points, TPL threads per line.
template <int N, int TPL = line_tl(N)>
struct FixedLine {
    static constexpr int kTl = TPL;
    static constexpr int kTx = TPL <= 32 ? 16 : TPL <= 48 ? 8 : TPL <= 256 ? 4 : 2;  // columns per block
    // threads of a block of rows: two short lines or more, or one of whole warps
    static constexpr int kRowT = TPL <= 32 ? 64 : TPL <= 64 || TPL == 128 ? 128 : TPL <= 256 ? 256 : 512;
    static constexpr bool kOne = TPL > line_tl(N);                                    // one group of points a thread
    static constexpr bool kLong = N > 5184;  // a full row's staged products do not fit beside the line
    using Inv = FixedLine<N, col_inv_tl(N)>;                                          // the inverse columns' line
    __host__ Inv inv() const { return Inv{tw}; }
    using Row = FixedLine<N, row_tl(N)>;                                               // the inverse rows' line
    __host__ Row row() const { return Row{tw}; }
    const float2* tw;
    // the same line with a twiddle pointer the compiler takes for a new one: a loop over lines then
    // reads its twiddles through L1 each time instead of hoisting dozens of them into spills
    __device__ __forceinline__ FixedLine fresh() const {
        FixedLine f = *this;
        asm volatile("" : "+l"(f.tw));
        return f;
    }
    __host__ __device__ __forceinline__ static constexpr int n() { return N; }
    __host__ __device__ __forceinline__ static constexpr int tl() { return TPL; }
    template <bool INV, bool LO = false, class In, class Out>
    __device__ __forceinline__ void run_io(float2* buf, int t, bool act, In&& in, Out&& out) const {
        mix_fft_io<N, TPL, INV, LO>(buf, tw, t, act && t < TPL, in, out);
    }
    template <bool INV, bool LO = false, class In>
    __device__ __forceinline__ void run_in(float2* buf, int t, bool act, In&& in) const {
        mix_fft_in<N, TPL, INV, LO>(buf, tw, t, act && t < TPL, in);
    }
};

}  // namespace zc
