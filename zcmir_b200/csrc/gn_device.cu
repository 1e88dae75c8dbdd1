// The batched Gauss–Newton refine on the device: the step, the candidate poses and the choice
// among them, so that a run of iterations needs no host round trip.
//
// Each iteration is, for n poses at once: the poses' inverse maps, their overlap moments,
// scores, tangent gradients and Gauss–Newton matrices (the pose kernels of pose.cu); then, one
// block per pose, the symmetric pair's gradient and matrix, the unit-ascent candidates (the step
// ladder `amps`) and the Gauss–Newton candidates (the solved step at 0.5, 1, 2, 4, 8 times, each
// capped at a tangent norm of 0.25), each composed onto the pose in normalised fixed
// coordinates; their scores; and, per pose, the first candidate in order that beats the score so
// far (by more than 1e-6 of it), as the host loop of the same search chooses. A pose that did
// not move is frozen. The pose algebra here restates the host's (lie.hpp, geom.hpp: the
// reference's src/lie.zig destN, hat, vee, expm3, projectGroup, composeN, adjointGrad,
// solveLinear) operation for operation in float64, and this file is compiled without fused
// multiply-adds, so the device loop and the host loop produce the same poses bit for bit.
#include <cuda_runtime.h>

#include "kernels.hpp"

namespace zc {
namespace {

// sums per pose row, tangent sums per pose row; candidates per pose: at most 16 ascent steps and
// the 5 Gauss–Newton multiples
constexpr int kMomN = 45, kGradN = 44, kMaxTry = 21;

__device__ void d_mul3(const double* a, const double* b, double* o) {
    double t[9];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) t[r * 3 + c] = a[r * 3] * b[c] + a[r * 3 + 1] * b[3 + c] + a[r * 3 + 2] * b[6 + c];
    for (int i = 0; i < 9; ++i) o[i] = t[i];
}

// inverse by the adjugate with one Newton refinement step (geom.hpp inv3)
__device__ void d_inv3(const double* m, double* o) {
    const double a = m[0], b = m[1], c = m[2], d = m[3], e = m[4], f = m[5], g = m[6], h = m[7], i = m[8];
    const double A = e * i - f * h, B = f * g - d * i, C = d * h - e * g;
    const double D = c * h - b * i, E = a * i - c * g, F = b * g - a * h;
    const double G = b * f - c * e, Hh = c * d - a * f, I = a * e - b * d;
    const double det = a * A + b * B + c * C;
    const double sg = det > 0 ? 1.0 : (det < 0 ? -1.0 : 0.0);
    const double s = 1.0 / (sg * fmax(fabs(det), 1e-18));
    const double inv[9] = {A * s, D * s, G * s, B * s, E * s, Hh * s, C * s, F * s, I * s};
    double p[9];
    d_mul3(m, inv, p);
    const double corr[9] = {2 - p[0], -p[1], -p[2], -p[3], 2 - p[4], -p[5], -p[6], -p[7], 2 - p[8]};
    d_mul3(inv, corr, o);
}

__device__ void d_destN(double w0, double h0, double* o) {
    const double w = fmax(w0, 1.0), h = fmax(h0, 1.0);
    const double sx = 0.5 * w, sy = 0.5 * h, cx = 0.5 * (w + 1), cy = 0.5 * (h + 1);
    const double v[9] = {1 / sx, 0, -cx / sx, 0, 1 / sy, -cy / sy, 0, 0, 1};
    for (int i = 0; i < 9; ++i) o[i] = v[i];
}

__device__ void d_hat(const double* x, bool homog, double* o) {
    double px = x[6], py = x[7], iso, z;
    if (!homog) {
        px = py = z = 0;
        iso = x[3];
    } else {
        iso = x[3] / 3;
        z = -2 * iso;
    }
    const double v[9] = {iso + x[4], x[5] - x[2], x[0], x[5] + x[2], iso - x[4], x[1], px, py, z};
    for (int i = 0; i < 9; ++i) o[i] = v[i];
}

__device__ void d_vee(const double* A0, bool homog, double* out) {
    double a = A0[0], e = A0[4];
    const double b = A0[1], c = A0[2], d = A0[3], f = A0[5], g = A0[6], h = A0[7], i = A0[8];
    if (homog) {
        const double tr = (a + e + i) / 3;
        a -= tr;
        e -= tr;
        const double iso = (a + e) / 2;
        const double v[8] = {c, f, (d - b) / 2, iso * 3, (a - e) / 2, (d + b) / 2, g, h};
        for (int k = 0; k < 8; ++k) out[k] = v[k];
        return;
    }
    const double v[8] = {c, f, (d - b) / 2, (a + e) / 2, (a - e) / 2, (d + b) / 2, 0, 0};
    for (int k = 0; k < 8; ++k) out[k] = v[k];
}

__device__ __forceinline__ double fin(double v) { return isfinite(v) ? v : 0.0; }

// one direction's gradient and Gauss–Newton matrix from its tangent sums (zero below 12 overlap)
__device__ void unpack(const double* t, double nsum, int nk, double* g, double* A) {
    for (int q = 0; q < 8; ++q) g[q] = 0;
    for (int q = 0; q < 64; ++q) A[q] = 0;
    if (!(nsum >= 12.0)) return;
    for (int q = 0; q < nk; ++q) g[q] = t[q];
    int h = 8;
    for (int q = 0; q < 8; ++q)
        for (int m = q; m < 8; ++m, ++h)
            if (q < nk && m < nk) A[q * nk + m] = A[m * nk + q] = t[h];
}

// the poses' inverse maps for the pose kernels: forward H⁻¹, inverse direction (H⁻¹)⁻¹
__global__ void k_gn_hinv(const double* __restrict__ H, int n, int sym, float* __restrict__ hinv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double Hi[9];
    d_inv3(H + (size_t)i * 9, Hi);
    for (int k = 0; k < 9; ++k) hinv[(size_t)i * 9 + k] = (float)Hi[k];
    if (sym) {
        double Hii[9];
        d_inv3(Hi, Hii);
        for (int k = 0; k < 9; ++k) hinv[((size_t)n + i) * 9 + k] = (float)Hii[k];
    }
}

// One element of a 3 × 3 product, in d_mul3's order.
__device__ __forceinline__ double mul3_at(const double* a, const double* b, int e) {
    const int r = 3 * (e / 3), c = e % 3;
    return a[r] * b[c] + a[r + 1] * b[3 + c] + a[r + 2] * b[6 + c];
}

// A block per pose. Each value is computed in the host loop's order by one thread, and values that do
// not depend on one another by threads of their own: the pull-back's 8 columns, the matrix's 64
// entries, the rows of the elimination, and the 9 entries of each candidate's 3 × 3 products (the
// exponential's series divides 117 entries a candidate). With a warp per pose and a lane per
// candidate the chains took 61 µs.
constexpr int kProposeThreads = 192;  // ≥ 9 · kMaxTry
static_assert(kProposeThreads >= 9 * kMaxTry, "nine threads per candidate");

__global__ void __launch_bounds__(kProposeThreads) k_gn_propose(GnDims d, GnAmps amps, const double* __restrict__ H,
                                                                const double* __restrict__ sums,
                                                                const double* __restrict__ score,
                                                                const double* __restrict__ tsum,
                                                                const unsigned char* __restrict__ active,
                                                                double* __restrict__ cur, double* __restrict__ Htry,
                                                                unsigned char* __restrict__ valid) {
    const int i = blockIdx.x, tid = threadIdx.x;
    const int T = d.T, nk = d.nk, n = d.n;
    const bool homog = d.homog != 0, sym = d.sym != 0;
    __shared__ double g[8], A[64], gf[8], Af[64], gb[8], Ab[64], PT[64], step[8], dv[8], cc[8][8], Mw[9], Mwi[9], N[9], Ni[9];
    __shared__ double M[64], rhs[8], fac[8], E[kMaxTry][9], P[kMaxTry][9], B[kMaxTry][9];
    __shared__ int use_ascent, use_step, piv, sq[kMaxTry];
    unsigned char* ok = valid + (size_t)i * T;
    if (tid < T) ok[tid] = 0;
    if (!active[i]) return;  // uniform over the block
    const double* Hp = H + (size_t)i * 9;
    // independent starts, a warp each: both directions' sums, the pull-back's map, the fixed frame
    if (tid == 0) {
        const double fwd = fin(score[i]), inv = sym ? fin(score[n + i]) : 0.0;
        cur[i] = sym ? 0.5 * (fwd + inv) : fwd;
        unpack(tsum + (size_t)i * kGradN, sums[(size_t)i * kMomN], nk, gf, Af);
    } else if (tid == 32 && sym) {
        unpack(tsum + ((size_t)n + i) * kGradN, sums[((size_t)n + i) * kMomN], nk, gb, Ab);
    } else if (tid == 64 && sym) {
        // M = N_moving H⁻¹ N_fixed⁻¹ and its inverse (lie.hpp adjoint_grad)
        double Hi[9], Nm[9], Nf[9], Nfi[9], t[9];
        d_inv3(Hp, Hi);
        d_destN(d.mw, d.mh, Nm);
        d_destN(d.fw, d.fh, Nf);
        d_inv3(Nf, Nfi);
        d_mul3(Nm, Hi, t);
        d_mul3(t, Nfi, Mw);
        d_inv3(Mw, Mwi);
    } else if (tid == 96) {
        d_destN(d.fw, d.fh, N);
        d_inv3(N, Ni);
    }
    __syncthreads();
    if (!sym) {
        if (tid < 64) A[tid] = Af[tid];
        if (tid < 8) g[tid] = gf[tid];
    } else {
        // tangent i through the pull-back: vee(M hat(e_i) M⁻¹)
        if (tid < nk) {
            double e[8] = {0, 0, 0, 0, 0, 0, 0, 0}, X[9], t[9];
            e[tid] = 1;
            d_hat(e, homog, X);
            d_mul3(Mw, X, t);
            d_mul3(t, Mwi, t);
            d_vee(t, homog, cc[tid]);
        }
        __syncthreads();
        if (tid < nk * nk) PT[tid] = 0.0 - cc[tid / nk][tid % nk];
        if (tid >= 64 && tid < 72) {
            const int q = tid - 64;
            double o = 0.0;
            if (q < nk)
                for (int j = 0; j < nk; ++j) o -= gb[j] * cc[q][j];
            g[q] = q < nk ? 0.5 * (gf[q] + o) : 0.0;
        }
        __syncthreads();
        if (tid < 64) A[tid] = 0;
        if (tid < nk * nk) {
            const int p = tid / nk, q = tid % nk;
            double s2 = 0;
            for (int x = 0; x < nk; ++x)
                for (int y = 0; y < nk; ++y) s2 += PT[p * nk + x] * Ab[x * nk + y] * PT[q * nk + y];
            A[tid] = 0.5 * (Af[tid] + s2);
        }
    }
    __syncthreads();
    // the unit ascent direction (src/lie.zig unitAscent); the Gauss–Newton system
    if (tid == 32) {
        use_ascent = 0;
        for (int q = 0; q < 8; ++q) dv[q] = 0;
        if (amps.n > 0) {
            double nr = 0;
            for (int q = 0; q < nk; ++q) dv[q] = g[q], nr += dv[q] * dv[q];
            nr = sqrt(nr);
            if (nr >= 1e-18)
                for (int q = 0; q < nk; ++q) dv[q] /= nr;
            double dn = 0;
            for (int q = 0; q < nk; ++q) dn += dv[q] * dv[q];
            use_ascent = sqrt(dn) > 1e-12;
        }
    }
    if (tid < nk * nk) M[tid] = A[tid] + (tid / nk == tid % nk ? 1e-4 * fmax(A[tid], 1e-12) : 0.0);
    if (tid < nk) rhs[tid] = 0.5 * g[tid];
    if (tid == 0) use_step = 1;
    __syncthreads();
    // M·step = rhs by Gauss–Jordan with partial pivoting (lie.hpp solve_linear); thread (r, c) one entry
    const int er = tid / nk, ec = tid % nk;
    for (int k = 0; k < nk; ++k) {
        if (tid == 0) {
            int b = k;
            for (int r = k + 1; r < nk; ++r)
                if (fabs(M[r * nk + k]) > fabs(M[b * nk + k])) b = r;
            piv = b;
        }
        __syncthreads();
        const int b = piv;
        if (b != k) {
            if (tid < nk) {
                const double t = M[k * nk + tid];
                M[k * nk + tid] = M[b * nk + tid];
                M[b * nk + tid] = t;
            } else if (tid == 32) {
                const double t = rhs[k];
                rhs[k] = rhs[b];
                rhs[b] = t;
            }
            __syncthreads();
        }
        const double dk = M[k * nk + k];
        if (!isfinite(dk) || fabs(dk) < 1e-300) {  // uniform over the block
            if (tid == 0) use_step = 0;
            break;
        }
        if (tid < nk) fac[tid] = tid == k ? 0.0 : M[tid * nk + k] / dk;
        __syncthreads();
        if (tid < nk * nk && er != k && ec >= k && fac[er] != 0) M[er * nk + ec] -= fac[er] * M[k * nk + ec];
        if (tid >= 64 && tid < 64 + nk && tid - 64 != k && fac[tid - 64] != 0) rhs[tid - 64] -= fac[tid - 64] * rhs[k];
        __syncthreads();
    }
    __syncthreads();
    if (tid < 8) step[tid] = (tid < nk && use_step) ? rhs[tid] / M[tid * nk + tid] : 0.0;
    __syncthreads();
    if (tid == 0 && use_step) {
        bool fine = true;
        for (int q = 0; q < nk; ++q) fine = fine && isfinite(step[q]);
        use_step = fine ? 1 : 0;
    }
    __syncthreads();
    // the candidates: the step ladder along the ascent direction, then the step's multiples (each
    // capped at a tangent norm of 0.25), as exp(ξ̂) in normalised fixed coordinates (lie.hpp composeN,
    // expm3: a 13-term Taylor series, scaled and squared)
    if (tid < T) {
        double x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        bool made = false;
        if (tid < amps.n) {
            if (use_ascent) {
                for (int k = 0; k < nk; ++k) x[k] = amps.v[tid] * dv[k];
                made = true;
            }
        } else if (use_step) {
            double nrm = 0;
            for (int q = 0; q < nk; ++q) nrm += step[q] * step[q];
            nrm = sqrt(nrm);
            const double mults[5] = {0.5, 1, 2, 4, 8};
            const double m = mults[tid - amps.n];
            const double sc = m * (nrm * m > 0.25 ? 0.25 / (nrm * m) : 1.0);
            for (int k = 0; k < nk; ++k) x[k] = sc * step[k];
            made = true;
        }
        double X[9], nrm = 0;
        d_hat(x, homog, X);
        for (int k = 0; k < 9; ++k) nrm = fmax(nrm, fabs(X[k]));
        int s = 0;
        for (double v = nrm; v > 0.5 && s < 10; v *= 0.5) ++s;
        const double sc = ldexp(1.0, -s);
        for (int k = 0; k < 9; ++k) {
            B[tid][k] = X[k] * sc;
            P[tid][k] = E[tid][k] = k % 4 == 0 ? 1.0 : 0.0;
        }
        sq[tid] = made ? s : -1;
    }
    __syncthreads();
    const int c = tid / 9, e = tid - 9 * c;
    const bool mine = c < T && sq[c < T ? c : 0] >= 0;
    for (int k = 1; k < 14; ++k) {
        const double v = mine ? mul3_at(P[c], B[c], e) / (double)k : 0.0;
        __syncthreads();
        if (mine) {
            P[c][e] = v;
            E[c][e] += v;
        }
        __syncthreads();
    }
    for (int k = 0; k < 10; ++k) {
        const bool go = mine && k < sq[c];
        if (!__syncthreads_or(go)) break;
        const double v = go ? mul3_at(E[c], E[c], e) : 0.0;
        __syncthreads();
        if (go) E[c][e] = v;
        __syncthreads();
    }
    // Ni E N H, then the group's normal form (projectGroup)
    if (mine) P[c][e] = mul3_at(Ni, E[c], e);
    __syncthreads();
    if (mine) E[c][e] = mul3_at(P[c], N, e);
    __syncthreads();
    if (mine) P[c][e] = mul3_at(E[c], Hp, e);
    __syncthreads();
    if (mine) {
        const double w = fabs(P[c][8]) > 1e-12 ? P[c][8] : 1;
        double v = P[c][e] / w;
        if (!homog && e >= 6) v = e == 8 ? 1 : 0;
        Htry[((size_t)i * T + c) * 9 + e] = v;
        if (e == 0) ok[c] = 1;
    }
}

// per pose, in candidate order, the first candidate that beats the score so far becomes the pose
__global__ void k_gn_select(GnDims d, const double* __restrict__ tscore, const unsigned char* __restrict__ valid,
                            const double* __restrict__ Htry, double* __restrict__ H, double* __restrict__ cur,
                            unsigned char* __restrict__ active) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const int T = d.T, nt = d.n * T;
    const bool sym = d.sym != 0;
    if (!active[i]) return;
    bool moved = false;
    double c = cur[i];
    for (int t = 0; t < T; ++t) {
        const size_t k = (size_t)i * T + t;
        if (!valid[k]) continue;
        const double fwd = fin(tscore[k]), inv = sym ? fin(tscore[nt + k]) : 0.0;
        const double s = sym ? 0.5 * (fwd + inv) : fwd;
        if (s > c + fmax(1e-6 * fabs(c), 1e-12)) {
            c = s;
            for (int q = 0; q < 9; ++q) H[(size_t)i * 9 + q] = Htry[k * 9 + q];
            moved = true;
        }
    }
    cur[i] = c;
    active[i] = moved ? 1 : 0;
}

}  // namespace

cudaError_t gn_hinv(const double* H, int n, int sym, float* hinv, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_gn_hinv<<<(n + 127) / 128, 128, 0, st>>>(H, n, sym, hinv);
    return cudaGetLastError();
}

cudaError_t gn_propose(const GnDims& d, const GnAmps& amps, const double* H, const double* sums, const double* score,
                       const double* tsum, const unsigned char* active, double* cur, double* Htry,
                       unsigned char* valid, cudaStream_t st) {
    if (d.n <= 0) return cudaSuccess;
    if (amps.n < 0 || amps.n > 16 || d.T != amps.n + 5 || d.T > kMaxTry) return cudaErrorInvalidValue;
    k_gn_propose<<<d.n, kProposeThreads, 0, st>>>(d, amps, H, sums, score, tsum, active, cur, Htry, valid);
    return cudaGetLastError();
}

cudaError_t gn_select(const GnDims& d, const double* tscore, const unsigned char* valid, const double* Htry, double* H,
                      double* cur, unsigned char* active, cudaStream_t st) {
    if (d.n <= 0) return cudaSuccess;
    k_gn_select<<<(d.n + 127) / 128, 128, 0, st>>>(d, tscore, valid, Htry, H, cur, active);
    return cudaGetLastError();
}

}  // namespace zc
