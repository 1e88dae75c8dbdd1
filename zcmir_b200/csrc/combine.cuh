// The per-shift SMI score, centred and whitened in float64 (the reference's combine_cell,
// shaders/smi.wgsl:825-915), shared by the row-pass kernels.
#pragma once

#include "box.cuh"
#include "kernels.hpp"

namespace zc {

// The correlation plan as compile-time tables (src/smi.zig:90-158): the moving and fixed plane
// of correlation c, and its slot in a plan that drops the fourth feature's planes.
__host__ __device__ constexpr int corr_a(int c) {
    return c == 0 ? 0 : c <= 4 ? c : c <= 8 ? 0 : c <= 24 ? 1 + (c - 9) / 4 : c <= 34 ? 5 + (c - 25) : 0;
}
__host__ __device__ constexpr int corr_b(int c) {
    return c <= 4 ? 0 : c <= 8 ? c - 4 : c <= 24 ? 1 + (c - 9) % 4 : c <= 34 ? 0 : 5 + (c - 35);
}
__host__ __device__ constexpr bool fourth_plane(int p) { return p == 4 || p == 8 || p == 11 || p == 13 || p == 14; }
__host__ __device__ constexpr bool corr_kept(int c, bool three) {
    return !three || (!fourth_plane(corr_a(c)) && !fourth_plane(corr_b(c)));
}
// Which correlations a map transforms: all of the plan (mode 0); without side A's moments over the
// fixed image's box (1: A's feature sums but the first and A's products); and without side B's over
// the moving image's box (2). Correlation 1 stays: it shares correlation 0's transforms.
__host__ __device__ constexpr bool corr_fft(int c, int mode) {
    return mode == 0 || !((c >= 2 && c <= 4) || (c >= 25 && c <= 34) || (mode == 2 && ((c >= 5 && c <= 8) || c >= 35)));
}
// Where correlation c's sum comes from, for every c: a slot of those kept and transformed (src 0), or
// a comp of side A's (1) or side B's (2) table, with n added back (diag). Tables rather than functions,
// so that a use at a compile-time c folds to a constant.
struct CorrSource {
    signed char src[45], at[45];
    bool diag[45];
};
template <int NF, int MODE>
__host__ __device__ constexpr CorrSource corr_source() {
    CorrSource t{};
    int slot = 0;
    for (int c = 0; c < 45; ++c) {
        t.src[c] = 0, t.at[c] = 0, t.diag[c] = false;
        if (!corr_kept(c, NF == 3)) continue;
        if (corr_fft(c, MODE)) {
            t.at[c] = (signed char)slot++;
            continue;
        }
        t.src[c] = c <= 4 || (c >= 25 && c <= 34) ? 1 : 2;
        if (c <= 8) {
            t.at[c] = (signed char)(c <= 4 ? c - 1 : c - 5);
        } else {
            const int k = c >= 35 ? c - 35 : c - 25, i = box_i(k, 4), j = box_j(k, 4);
            t.at[c] = (signed char)box_comp(i, j, NF);
            t.diag[c] = i == j;
        }
    }
    return t;
}

// how many slots a map of the given plan transforms (NF = 1: the NCC map's one)
template <int NF, bool EXACT, int MODE>
__host__ __device__ constexpr int corr_slots() {
    if (NF == 1) return 1;
    int n = 0;
    for (int c = 0; c < (EXACT ? 45 : 25); ++c) n += corr_kept(c, NF == 3) && corr_fft(c, MODE) ? 1 : 0;
    return n;
}

__host__ __device__ constexpr int tri_kc(int i, int j) {
    return (i < j ? i : j) * 4 - ((i < j ? i : j) * ((i < j ? i : j) + 1)) / 2 + (i < j ? j : i);
}

// the correlation area where it lives in device memory
__device__ __forceinline__ void read_area(CombineParams& cp) {
    if (cp.area_dev) cp.area = *cp.area_dev;
}

// The score's parameters for the shifts of row y of an ny-row map: a log-polar map scales row
// y's sums by e^{kΔλ}·Δλ·Δθ (k the row's wrapped log-radius lag, smi.wgsl:777-795 extract_pair).
__device__ __forceinline__ CombineParams row_params(const CombineParams& cp, int y, int ny) {
    CombineParams r = cp;
    if (cp.lp_dlam != 0.0) {
        const int k = y <= ny / 2 ? y : y - ny;
        r.inv_nn = cp.inv_nn * exp((double)k * cp.lp_dlam) * cp.lp_dlam * cp.lp_dth;
    }
    return r;
}
// the zero-lag overlap in the map's units (row 0 of a log-polar map carries Δλ·Δθ)
__device__ __forceinline__ double lag0_units(const CombineParams& cp, double n00) {
    return cp.lp_dlam != 0.0 ? n00 * cp.lp_dlam * cp.lp_dth : n00;
}

// Whether a shift's overlap n is above the floors (else its score is 0; a NaN overlap is not below).
template <bool CALIB>
__device__ __forceinline__ bool overlap_alive(double n, const CombineParams& p, double n00) {
    const double floor_n = CALIB ? (double)p.min_n : fmax((double)p.min_n, 0.08 * fmax(n00, 0.0));
    return !(n < floor_n || (CALIB && n / fmax(p.area, 1.0) <= 10.0));
}

// Per-shift score (smi.wgsl:825-915, combine_cell): centring, ridge, Cholesky factors and the
// whitened norm in float64, the calibrated map's Wilson–Hilferty transform in float32; every
// index known at compile time (NF features, exact or global whitening, calibrated or not), so the 4×4
// algebra stays in registers. n: this shift's overlap, above the floors (overlap_alive); `mean(c, 1 / n)`
// returns correlation c's sum over n (of the 45; NF = 3 asks for none of the fourth feature's), and every c
// passed to it is a compile-time constant. Each Cholesky pivot is inverted once (rsqrt) and the
// substitutions multiply by it.
template <int NF, bool EXACT, bool CALIB, class G>
__device__ __forceinline__ float combine_smi(G&& mean, double n, const CombineParams& p) {
    const double neff = n / fmax(p.area, 1.0);
    const double rn = 1.0 / fmax(n, 1e-8);
    auto S = [&](int c) -> double { return mean(c, rn); };
    double ma[NF], mb[NF], C[NF][NF];
#pragma unroll
    for (int i = 0; i < NF; ++i) {
        ma[i] = S(1 + i);
        mb[i] = S(5 + i);
    }
#pragma unroll
    for (int i = 0; i < NF; ++i)
#pragma unroll
        for (int j = 0; j < NF; ++j) C[i][j] = S(9 + 4 * i + j) - ma[i] * mb[j];
    if (!EXACT) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < NF; ++i)
#pragma unroll
            for (int j = 0; j < NF; ++j) {
                const double c = fmin(fmax(C[i][j], -1.0), 1.0);
                s += c * c;
            }
        const double sc = n * s;
        return (sc == sc) ? (float)sc : 0.f;
    }
    double A[NF][NF], B[NF][NF];
    double tra = 0.0, trb = 0.0;
#pragma unroll
    for (int i = 0; i < NF; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            A[i][j] = S(25 + tri_kc(i, j)) - ma[i] * ma[j];
            B[i][j] = S(35 + tri_kc(i, j)) - mb[i] * mb[j];
        }
        tra += A[i][i];
        trb += B[i][i];
    }
    const double rga = p.ridge * fmax(tra * 0.25, 1e-12), rgb = p.ridge * fmax(trb * 0.25, 1e-12);
    double ia[NF], ib[NF];  // 1 / L_ii
#pragma unroll
    for (int i = 0; i < NF; ++i) {
        A[i][i] += rga;
        B[i][i] += rgb;
    }
#pragma unroll
    for (int i = 0; i < NF; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double sa = A[i][j], sb = B[i][j];
#pragma unroll
            for (int k = 0; k < j; ++k) {
                sa -= A[i][k] * A[j][k];
                sb -= B[i][k] * B[j][k];
            }
            if (i == j) {
                if (!(sa > 0.0) || !(sb > 0.0)) return 0.f;
                ia[i] = rsqrt(sa);
                ib[i] = rsqrt(sb);
                A[i][i] = sa * ia[i];
                B[i][i] = sb * ib[i];
            } else {
                A[i][j] = sa * ia[j];
                B[i][j] = sb * ib[j];
            }
        }
    }
    // X = L_A⁻¹ C (forward substitution down each column), in place in C
#pragma unroll
    for (int j = 0; j < NF; ++j)
#pragma unroll
        for (int i = 0; i < NF; ++i) {
            double s = C[i][j];
#pragma unroll
            for (int k = 0; k < i; ++k) s -= A[i][k] * C[k][j];
            C[i][j] = s * ia[i];
        }
    // Y = X L_B⁻ᵀ row by row, ‖Y‖² as it goes
    double acc = 0.0;
#pragma unroll
    for (int r = 0; r < NF; ++r) {
        double yv[NF];
#pragma unroll
        for (int i = 0; i < NF; ++i) {
            double s = C[r][i];
#pragma unroll
            for (int k = 0; k < i; ++k) s -= B[i][k] * yv[k];
            yv[i] = s * ib[i];
            acc += yv[i] * yv[i];
        }
    }
    double score = n * acc;
    if (CALIB) {
        // the Wilson–Hilferty transform of the whitened statistic in float32: the float64 steps
        // are the centring and the Cholesky factors above; this tail only rescales their result
        constexpr float q = NF;
        const float v = fminf((float)acc, q - 1e-4f);
        const float nq = (float)neff - q - 1.0f;
        const float fv = nq * v / (q * (q - v));
        constexpr float a = 2.0f / (9.0f * q * q);
        const float b = 2.0f / (9.0f * q * nq);
        const float cc = cbrtf(fmaxf(fv, 0.0f));
        const float z = ((1.0f - b) * cc - (1.0f - a)) * rsqrtf(b * cc * cc + a);
        score = fmaxf(z, 0.0f);
    }
    return (score == score) ? (float)score : 0.f;
}

// The NCC map's value at a lag (src/overlay.zig:256-258): the mean-free correlation over the
// product of the planes' norms (den, carried in the n00 slot), clamped to ±1.5.
__device__ __forceinline__ float combine_ncc(double sum, double den) {
    return (float)fmin(1.5, fmax(-1.5, sum / den));
}

// A shift whose sums are all transformed ones: raw(c) the unscaled float sum of correlation c. NF = 1
// selects the NCC map, 3 or 4 the SMI score over that many features.
template <int NF, bool EXACT, bool CALIB, class G>
__device__ __forceinline__ float combine_t(G&& raw, const CombineParams& p, double n00) {
    const double n = (double)raw(0) * p.inv_nn;
    if constexpr (NF == 1) {
        return combine_ncc(n, n00);
    } else {
        if (!overlap_alive<CALIB>(n, p, n00)) return 0.f;
        double scale = 0.0;  // inv_nn / n, once per shift
        bool have = false;
        return combine_smi<NF, EXACT, CALIB>(
            [&](int c, double rn) -> double {
                if (!have) scale = p.inv_nn * rn, have = true;
                return (double)raw(c) * scale;
            },
            n, p);
    }
}

}  // namespace zc
