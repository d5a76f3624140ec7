// ss_regular.cu — regularGridTransform on the device for RL and RLZ grids
// (src/transforms_cylindrical.jl:929-1020 RL, 1168-1287 RLZ): the spectral
// array evaluated on a tensor-product (r, λ[, z]) point set.
//
//   reg_sa        SAtransform! of every spectral slot (each Chebyshev mode, each
//                 wavenumber's cos / sin block), FP64, the grid's spline factor
//   reg_si        SI / SIx / SIxx of those coefficients at the r points
//   reg_fourier   the Fourier series at the λ points with the R2HC half-amplitude
//                 factor 2: f, ∂r f, ∂rr f (from SI, SIx, SIxx) and ∂λ f, ∂λλ f
//   reg_cheb      (RLZ) CAtransform! and the Chebyshev series at the z points, as
//                 per-variable matrices composed on the host: value for every
//                 variant, ∂z and ∂zz for the value variant
// Every stage computes in FP64 whatever the grid's precision; the result is a
// host array (n_r·n_λ[·n_z], nvars, 5|7), λ (then z) fastest, as the reference
// returns it.  The reference runs SAtransform! on the grid's spline objects,
// whose R3X background (ahat) is zero unless multipatch coupling set it; this
// path applies no ahat.
#include <cuda_runtime.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <utility>
#include <vector>

#include "ss_grid.h"
#include "ss_kernels.h"
#include "ss_spline_dev.cuh"
#include "ss_types.cuh"

using namespace ss;

#define CUDA_TRY(expr)                                                                      \
    do {                                                                                    \
        cudaError_t _e = (expr);                                                            \
        if (_e != cudaSuccess) {                                                            \
            set_error("%s failed: %s", #expr, cudaGetErrorString(_e));                      \
            return (_e == cudaErrorMemoryAllocation) ? SS_OUT_OF_MEMORY : SS_CUDA_ERROR;   \
        }                                                                                   \
    } while (0)

namespace {

// SAtransform! of `per` consecutive slots of one item per CTA (one thread each):
// Γ fold, banded LLᵀ solve with the FP64 factor, Γᵀ unfold → coef[item][slot][b]
template <typename P>
__global__ void reg_sa_kernel(const P *spec, const SplineDev *spl, double *coef, int64_t nspec, int b, int ld,
                              int nslots_z, int bk) {
    extern __shared__ __align__(16) double sm[];
    const int item = blockIdx.y, v = item / bk, zb = item % bk;
    const SplineDev &sp = spl[v];
    const int n = sp.Min, per = blockDim.x;
    double *X = sm;              // per × ld
    double *Ls = X + per * ld;   // 4n
    double *Di = Ls + 4 * n;     // n
    const int s0 = blockIdx.x * per, nsl = min(per, nslots_z - s0);
    const P *src = spec + (size_t)v * nspec + ((size_t)zb * nslots_z + s0) * b;
    for (int e = threadIdx.x; e < nsl * b; e += per) X[(e / b) * ld + e % b] = (double)src[e];
    for (int e = threadIdx.x; e < 4 * n; e += per) Ls[e] = sp.L4[e];
    for (int e = threadIdx.x; e < n; e += per) Di[e] = sp.dinv[e];
    __syncthreads();
    if (threadIdx.x < nsl) {
        double *x = X + threadIdx.x * ld;
        gamma_fold(sp, x, b, n);
        band_solve(Ls, Di, x, n, sp.periodic ? sp.tail : nullptr);
        gamma_unfold(sp, x, b, n);
    }
    __syncthreads();
    double *dst = coef + ((size_t)item * nslots_z + s0) * b;
    for (int e = threadIdx.x; e < nsl * b; e += per) dst[e] = X[(e / b) * ld + e % b];
}

// sr[d][item][r][slot] = Σ_tap w[d][r][tap] · coef[item][slot][m0[r] + tap]
__global__ void reg_si_kernel(const double *coef, const int *m0, const double *w, double *sr, int b,
                              int nslots_z, int n_r, int nitems) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y, item = blockIdx.z;
    if (s >= nslots_z) return;
    const double *a = coef + ((size_t)item * nslots_z + s) * b + m0[r];
    const double a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double *wd = w + ((size_t)d * n_r + r) * 4;
        sr[(((size_t)d * nitems + item) * n_r + r) * nslots_z + s] = wd[0] * a0 + wd[1] * a1 + wd[2] * a2 + wd[3] * a3;
    }
}

// ---- cos(kλ), sin(kλ) tables
// π/2 in parts of 33, 33 and 53 bits (reduction after Cody and Waite 1980)
constexpr double kPio2a = 0x1.921fb54400000p+0, kPio2b = 0x1.0b4611a600000p-34, kPio2c = 0x1.3198a2e037073p-69;
// cos and sin of a, |a| < 2^20: a − n·π/2 in two words (n times the first two parts is
// exact), then the Taylor series with the leading terms in two words.  Against 64-bit
// significands: 0.59 units of the last place at most and 0.288 rms over 4 million k·λ with
// k ≤ 10^5, as the host library's 0.288 (cos and sin of the CUDA library: 0.36).
__device__ __forceinline__ void cos_sin_accurate(double a, double &c, double &s) {
    const double n = rint(a * 0.63661977236758134);
    const double t = fma(-n, kPio2a, a);
    const double m = n * kPio2b;
    double h = t - m, v = t - h;
    double l = fma(-n, kPio2c, (t - (h + v)) + (v - m));
    const double h1 = h + l;  // renormalised
    l = l - (h1 - h);
    h = h1;
    const double z = h * h, zl = fma(h, h, -z) + 2.0 * (h * l);
    // sin: h − h³/6 + h⁵/120 − …
    const double w = h * z, wl = fma(h, z, -w) + fma(h, zl, l * z);
    const double k3 = 1.0 / 6.0, k3l = fma(-k3, 6.0, 1.0) / 6.0;
    const double g = w * k3, gl = fma(w, k3, -g) + fma(w, k3l, wl * k3);
    double p = -1.0 / 121645100408832000.0;
    p = fma(p, z, 1.0 / 355687428096000.0);
    p = fma(p, z, -1.0 / 1307674368000.0);
    p = fma(p, z, 1.0 / 6227020800.0);
    p = fma(p, z, -1.0 / 39916800.0);
    p = fma(p, z, 1.0 / 362880.0);
    p = fma(p, z, -1.0 / 5040.0);
    p = fma(p, z, 1.0 / 120.0);
    const double u = h - g;
    const double sn = u + (((h - u) - g) + (fma(w * z, p, l - gl)));
    // cos: 1 − h²/2 + h⁴/24 − …
    double q = -1.0 / 6402373705728000.0;
    q = fma(q, z, 1.0 / 20922789888000.0);
    q = fma(q, z, -1.0 / 87178291200.0);
    q = fma(q, z, 1.0 / 479001600.0);
    q = fma(q, z, -1.0 / 3628800.0);
    q = fma(q, z, 1.0 / 40320.0);
    q = fma(q, z, -1.0 / 720.0);
    q = fma(q, z, 1.0 / 24.0);
    const double y = 1.0 - 0.5 * z;
    const double cn = y + (((1.0 - y) - 0.5 * z) + fma(z * z, q, -0.5 * zl));
    const int k = (int)n & 3;
    const double cc = (k & 1) ? sn : cn, ss = (k & 1) ? cn : sn;
    c = (k == 1 || k == 2) ? -cc : cc;
    s = k >= 2 ? -ss : ss;
}
constexpr double kRegMaxAngle = 1e6;  // bound of kλ for the tables above
// tc, ts[(k−1)·n_λ + j] of the rounded products kλ_j, as on the host: K = 180 × 361 points
// took 1.2 ms there, two thirds of the time before the first launch
__global__ void __launch_bounds__(128) reg_table_kernel(const double *lam, double *tc, double *ts, int K, int n_lam) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= (int64_t)K * n_lam) return;
    cos_sin_accurate((double)(e / n_lam + 1) * lam[e % n_lam], tc[e], ts[e]);
}

// The Fourier series at λ_j for one (item, r) per CTA row, j over threads:
//   f = a0 + Σ_k 2 (rc cos kλ + rs sin kλ), the same with the SIx / SIxx
//   coefficients for ∂r f / ∂rr f, ∂λ f = Σ_k 2k (−rc sin + rs cos),
//   ∂λλ f = −Σ_k 2k² (rc cos + rs sin)   (src/transforms_cylindrical.jl:985-1005)
// cos/sin(kλ_j) come from the tables tc/ts[(k−1)·n_λ + j].  RL writes the result
// slots straight into out (rows r·n_λ + j); RLZ writes fb[variant][v][r][j][zb].
// Bound by binary64 operations (two multiply-adds a clock and SM): the factors 2, 2k
// and 2k² go into the coefficients as they are staged, once per CTA, which leaves ten
// multiply-adds per (k, λ) where the sums above take sixteen operations and an integer
// conversion.  Cosine and sine terms are summed apart: one rounding of each sum per k, as
// many as the paired sum has (in one sum the error grows 1.4 times), and each chunk apart
// (error of sums of 20 to 720 random terms: 0.4 of the paired sum's).  61 × 361 columns
// of 32 modes, K = 180: 4.16 → 2.25 ms (the operations alone 2.2 ms).  A chunk is kRegChunk
// wavenumbers, 5 KB of staged coefficients.
constexpr int kRegChunk = 64;
__global__ void __launch_bounds__(128) reg_fourier_kernel(const double *sr, const double *tc, const double *ts,
                                                          double *dst, int nslots_z, int K, int n_r, int n_lam,
                                                          int nitems, int rlz, int bk, int nvars) {
    // per k: f, ∂r, ∂rr, ∂λ, ∂λλ as (factor of cos, factor of sin)
    __shared__ __align__(16) double2 c[kRegChunk][5];
    const int r = blockIdx.y, item = blockIdx.z;
    const size_t ds = (size_t)nitems * n_r * nslots_z;
    const double *c0 = sr + ((size_t)item * n_r + r) * nslots_z, *c1 = c0 + ds, *c2 = c1 + ds;
    const int j = blockIdx.x * blockDim.x + threadIdx.x, jj = min(j, n_lam - 1);
    double vals[5] = {c0[0], c1[0], c2[0], 0.0, 0.0};  // variants: f, ∂r, ∂rr, ∂λ, ∂λλ
    for (int k0 = 1; k0 <= K; k0 += kRegChunk) {
        const int nk = min(kRegChunk, K + 1 - k0);
        __syncthreads();
        for (int q = threadIdx.x; q < nk; q += blockDim.x) {
            const int k = k0 + q;
            const double kk = 2.0 * (double)k, k2 = -(kk * (double)k);
            const double rc = c0[2 * k - 1], rs = c0[2 * k];
            c[q][0] = make_double2(2.0 * rc, 2.0 * rs);
            c[q][1] = make_double2(2.0 * c1[2 * k - 1], 2.0 * c1[2 * k]);
            c[q][2] = make_double2(2.0 * c2[2 * k - 1], 2.0 * c2[2 * k]);
            c[q][3] = make_double2(kk * rs, -kk * rc);
            c[q][4] = make_double2(k2 * rc, k2 * rs);
        }
        __syncthreads();
        const double *pc = tc + (size_t)(k0 - 1) * n_lam + jj, *ps = ts + (size_t)(k0 - 1) * n_lam + jj;
        if (j < n_lam) {
            double u[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, w[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // cos and sin sums
            for (int q = 0; q < nk; q++, pc += n_lam, ps += n_lam) {
                const double ck = *pc, sk = *ps;
                u[0] = fma(c[q][0].x, ck, u[0]);
                w[0] = fma(c[q][0].y, sk, w[0]);
                u[1] = fma(c[q][1].x, ck, u[1]);
                w[1] = fma(c[q][1].y, sk, w[1]);
                u[2] = fma(c[q][2].x, ck, u[2]);
                w[2] = fma(c[q][2].y, sk, w[2]);
                u[3] = fma(c[q][3].x, ck, u[3]);
                w[3] = fma(c[q][3].y, sk, w[3]);
                u[4] = fma(c[q][4].x, ck, u[4]);
                w[4] = fma(c[q][4].y, sk, w[4]);
            }
#pragma unroll
            for (int q = 0; q < 5; q++) vals[q] += u[q] + w[q];
        }
    }
    if (j >= n_lam) return;
    if (!rlz) {
        const size_t nrows = (size_t)n_r * n_lam, row = (size_t)r * n_lam + j;
#pragma unroll
        for (int q = 0; q < 5; q++) dst[((size_t)q * nvars + item) * nrows + row] = vals[q];
    } else {
        const int v = item / bk, zb = item - v * bk;
#pragma unroll
        for (int q = 0; q < 5; q++)
            dst[((((size_t)q * nvars + v) * n_r + r) * n_lam + j) * bk + zb] = vals[q];
    }
}

// Chebyshev series at z for every (r, λ) column of one variable and variant:
// out[row = col·n_z + z][v][slot] = Σ_zb M[z][zb] fb[col][zb], M = E·CA (value),
// and for the value variant also Dz·CA (∂z) and Dzz·CA (∂zz)
__global__ void reg_cheb_kernel(const double *fb, const double *mats, double *out, int64_t ncol, int n_z, int bk,
                                int nvars, int n_r) {
    extern __shared__ __align__(16) double M[];  // 3 × n_z × bk
    const int v = blockIdx.y, q = blockIdx.z;
    const int nm = (q == 0) ? 3 : 1;
    const double *mv = mats + (size_t)v * 3 * n_z * bk;
    for (int e = threadIdx.x; e < nm * n_z * bk; e += blockDim.x) M[e] = mv[e];
    __syncthreads();
    const int64_t nrows = ncol * n_z;
    const double *src = fb + ((size_t)q * nvars + v) * ncol * bk;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nrows; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t col = t / n_z;
        const int z = (int)(t - col * n_z);
        const double *bcol = src + col * bk;
        for (int m = 0; m < nm; m++) {
            const double *row = M + ((size_t)m * n_z + z) * bk;
            double acc = 0.0;
            for (int i = 0; i < bk; i++) acc += row[i] * bcol[i];
            const int slot = m == 0 ? q : 4 + m;  // variant q's slot; ∂z, ∂zz → slots 6, 7 (0-based 5, 6)
            out[((size_t)slot * nvars + v) * nrows + t] = acc;
        }
    }
    (void)n_r;
}

// Value of the spectral fields at arbitrary points: one warp per (point, variable).
// Per Chebyshev mode z_b the warp sums the Fourier series of the SI values at the
// point's radius (4-tap window m0, weights w):
//   f_zb = S_0 + 2 Σ_k (S_{2k−1} cos kλ + S_{2k} sin kλ),  S_q = Σ_tap w_tap a_q[m0 + tap]
// (src/interpolation.jl:1628-1656 RL, 1670-1718 RLZ).  mode 1 keeps the k = 0
// term only (the azimuthal mean), mode 2 writes NaN; taper t blends
// t·full + (1 − t)·mean (src/relocation.jl:252-258).  RL: one value per point.
// RLZ: CAtransform! of f_zb (the composed matrix CA, N × bk) and the Chebyshev
// series at z (_cheb_eval_single, src/interpolation.jl:1271-1285) — at the
// point's own z (zcol = nullptr) or at the n_z column levels zcol (relocation).
struct PointArgs {
    const double *coef;   // [item][slot][b] spline coefficients (FP64)
    const double *lam, *z, *w, *taper;  // per point; z RLZ only; w[p][4]
    const int *m0, *mode;
    const double *ca;     // RLZ: per variable N × bk
    const double *zcol;   // RLZ relocation: n_z column levels, else null
    void *out;            // P storage
    int64_t npts, ostride_v;  // rows between variables of out
    int b, nslots, K, bk, nvars, N, n_z, rlz, out_f32;
    double zmin, zmax;
    int first_var, nvar_eval;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(128) point_eval_kernel(PointArgs A) {
    extern __shared__ __align__(16) double fz[];  // per warp: bk values
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    const int64_t p = gw / A.nvar_eval;
    if (p >= A.npts) return;  // whole warps leave together (no block barrier below)
    const int v = A.first_var + (int)(gw - p * A.nvar_eval);
    double *f = fz + (size_t)wib * A.bk;
    const int mode = A.mode ? A.mode[p] : 0;
    auto store = [&](int64_t row, double val) {
        if (A.out_f32) ((float *)A.out)[(size_t)v * A.ostride_v + row] = (float)val;
        else ((double *)A.out)[(size_t)v * A.ostride_v + row] = val;
    };
    const int nout = A.rlz && A.zcol ? A.n_z : 1;
    const int64_t row0 = A.rlz && A.zcol ? p * A.n_z : p;
    if (mode == 2) {
        if (lane < nout) store(row0 + lane, __longlong_as_double(0x7ff8000000000000LL));
        for (int q = lane + 32; q < nout; q += 32) store(row0 + q, __longlong_as_double(0x7ff8000000000000LL));
        return;
    }
    const double lam = A.lam[p], t = A.taper ? A.taper[p] : 1.0;
    const double w0 = A.w[p * 4], w1 = A.w[p * 4 + 1], w2 = A.w[p * 4 + 2], w3 = A.w[p * 4 + 3];
    const int m0 = A.m0[p];
    for (int zb = 0; zb < A.bk; zb++) {
        const double *a = A.coef + ((size_t)(v * A.bk + zb) * A.nslots) * A.b + m0;
        auto si = [&](int q) {
            const double *c = a + (size_t)q * A.b;
            return w0 * c[0] + w1 * c[1] + w2 * c[2] + w3 * c[3];
        };
        double full = 0.0;
        if (mode == 0)
            for (int k = 1 + lane; k <= A.K; k += 32) {
                double sk, ck;
                sincos((double)k * lam, &sk, &ck);
                full += 2.0 * (si(2 * k - 1) * ck + si(2 * k) * sk);
            }
        full = warp_sum(full);
        const double mean = si(0);
        const double val = (mode == 1) ? mean : (t * (mean + full) + (1.0 - t) * mean);
        if (lane == 0) f[zb] = val;
    }
    __syncwarp();
    if (!A.rlz) {
        if (lane == 0) store(p, f[0]);
        return;
    }
    // CAtransform! then the Chebyshev series (clamped to [−1, 1]) at each level
    const double scale = -0.5 * (A.zmax - A.zmin), offset = 0.5 * (A.zmin + A.zmax);
    const double *ca = A.ca + (size_t)v * A.N * A.bk;
    for (int zi = 0; zi < nout; zi++) {
        const double z = A.zcol ? A.zcol[zi] : A.z[p];
        const double xi = fmin(fmax((z - offset) / scale, -1.0), 1.0);
        const double th = acos(xi);
        double acc = 0.0;
        for (int n = lane; n < A.N; n += 32) {
            double an = 0.0;
            for (int i = 0; i < A.bk; i++) an += ca[(size_t)n * A.bk + i] * f[i];
            const double e = (n == 0) ? 1.0 : (n == A.N - 1 ? cos((double)n * th) : 2.0 * cos((double)n * th));
            acc += e * an;
        }
        acc = warp_sum(acc);
        if (lane == 0) store(row0 + zi, acc);
    }
}

// E (value), Dz, Dzz of the DCT-I series at z (n_z × N, row-major) with the
// reference's clamps (_cheb_eval_pts!, _cheb_dz_pts!, _cheb_dzz_pts!,
// src/transforms_cylindrical.jl:1030-1094)
void cheb_point_matrices(int N, double zmin, double zmax, const double *z, int n_z, std::vector<double> &E,
                         std::vector<double> &Dz, std::vector<double> &Dzz) {
    const double scale = -0.5 * (zmax - zmin), offset = 0.5 * (zmin + zmax);
    E.assign(size_t(n_z) * N, 0.0);
    Dz.assign(size_t(n_z) * N, 0.0);
    Dzz.assign(size_t(n_z) * N, 0.0);
    for (int i = 0; i < n_z; i++) {
        const double xi0 = std::min(std::max((z[i] - offset) / scale, -1.0 + 1e-14), 1.0 - 1e-14);
        const double t0 = std::acos(xi0);
        const double xi = std::min(std::max((z[i] - offset) / scale, -1.0 + 1e-10), 1.0 - 1e-10);
        const double t = std::acos(xi), st = std::sin(t), ct = std::cos(t);
        for (int k = 0; k < N; k++) {
            const double m = (double)k;
            const double wgt = (k == 0) ? 0.0 : (k == N - 1 ? 1.0 : 2.0);
            E[size_t(i) * N + k] = (k == 0) ? 1.0 : (k == N - 1 ? std::cos(m * t0) : 2.0 * std::cos(m * t0));
            const double d1 = -wgt * m * std::sin(m * t);       // df/dt coefficient
            const double d2 = -wgt * m * m * std::cos(m * t);   // d²f/dt² coefficient
            Dz[size_t(i) * N + k] = d1 / (-scale * st);
            Dzz[size_t(i) * N + k] = (d2 * st - d1 * ct) / (scale * scale * st * st * st);
        }
    }
}

// The device buffers of one regularGridTransform call: the grid's kept block if it is
// there and large enough, else a new one.  A call takes the block out, so calls on several
// threads or streams never share it, and puts back the larger one after its stream has
// drained; blocks above kRegKeep are freed.  (Nine allocations and frees took 75 to 240 µs
// of a call on 39 × 157 × 13 points, by the state of the allocator.)
constexpr size_t kRegKeep = (size_t)256 << 20;
struct RegBlock {
    ss_grid *g;
    void *p = nullptr;
    size_t bytes = 0;
    cudaError_t e = cudaSuccess;
    RegBlock(ss_grid *grid, size_t need) : g(grid) {
        {
            std::lock_guard<std::mutex> lock(g->reg_mutex);
            std::swap(p, g->reg_block);
            std::swap(bytes, g->reg_bytes);
        }
        if (bytes >= need) return;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = std::max<size_t>(need, 256);
        e = cudaMalloc(&p, bytes);
        if (e != cudaSuccess) { p = nullptr; bytes = 0; }
    }
    ~RegBlock() {
        if (bytes <= kRegKeep) {
            std::lock_guard<std::mutex> lock(g->reg_mutex);
            if (bytes > g->reg_bytes) {
                std::swap(p, g->reg_block);
                std::swap(bytes, g->reg_bytes);
            }
        }
        if (p) cudaFree(p);
    }
    RegBlock(const RegBlock &) = delete;
    RegBlock &operator=(const RegBlock &) = delete;
};

template <typename P>
int32_t regular(ss_grid *g, const double *r_pts, int n_r, const double *lam_pts, int n_lam, const double *z_pts,
                int n_z, double *out_host, cudaStream_t st) {
    const ss_dims &d = g->d;
    const int b = (int)d.b_iDim, K = (int)d.kDim_wn, ns = g->nslots_z, bk = (int)d.b_kDim;
    const int nv = (int)d.nvars, nitems = g->nitems;
    const int nz = g->rlz ? n_z : 1;
    const size_t nrows = size_t(n_r) * n_lam * nz;
    // host tables: SI weights at r, cos/sin(kλ), Chebyshev point matrices composed with CA
    std::vector<int> m0;
    std::vector<double> w;
    spline_point_weights(g->spl_host[0], r_pts, n_r, m0, w);  // every variable shares the radial knots
    bool dev_tables = true;  // large, infinite and NaN points: the host's tables
    for (int j = 0; j < n_lam; j++) dev_tables &= std::fabs(lam_pts[j]) * K < kRegMaxAngle;
    std::vector<double> tc(dev_tables ? 0 : size_t(K) * n_lam), ts(tc.size());
    for (int k = 1; k <= K && !dev_tables; k++)
        for (int j = 0; j < n_lam; j++) {
            const double a = (double)k * lam_pts[j];
            tc[size_t(k - 1) * n_lam + j] = std::cos(a);
            ts[size_t(k - 1) * n_lam + j] = std::sin(a);
        }
    std::vector<double> mats;
    if (g->rlz) {
        const int N = (int)d.kDim;
        std::vector<double> E, Dz, Dzz;
        cheb_point_matrices(N, g->p.kMin, g->p.kMax, z_pts, n_z, E, Dz, Dzz);
        mats.assign(size_t(nv) * 3 * n_z * bk, 0.0);
        for (int v = 0; v < nv; v++) {
            ChebHost ch;
            int32_t rc = build_cheb(N, bk, g->bcb[v], g->bct[v], g->p.kMin, g->p.kMax, ch);
            if (rc) return rc;
            // CA[n][i] = δ_ni + Σ_p v_p[n] u_p[i]  (a = bfill + Γᵀ bfill)
            std::vector<double> CA(size_t(N) * bk, 0.0);
            for (int n = 0; n < N; n++)
                for (int i = 0; i < bk; i++) {
                    double a = (n == i) ? 1.0 : 0.0;
                    for (int p = 0; p < ch.nrank; p++) a += ch.gv[size_t(p) * N + n] * ch.gu[size_t(p) * bk + i];
                    CA[size_t(n) * bk + i] = a;
                }
            const std::vector<double> *src[3] = {&E, &Dz, &Dzz};
            for (int m = 0; m < 3; m++)
                for (int z = 0; z < n_z; z++)
                    for (int i = 0; i < bk; i++) {
                        double acc = 0.0;
                        for (int n = 0; n < N; n++) acc += (*src[m])[size_t(z) * N + n] * CA[size_t(n) * bk + i];
                        mats[((size_t(v) * 3 + m) * n_z + z) * bk + i] = acc;
                    }
        }
    }
    // device buffers: one block, kept by the grid for its next call
    const size_t out_elems = nrows * nv * d.nslots;
    const size_t need[9] = {size_t(nitems) * ns * b * 8, w.size() * 8, m0.size() * 4, (size_t(K) + 1) * n_lam * 8, size_t(K) * n_lam * 8,
                            size_t(3) * nitems * n_r * ns * 8, out_elems * 8,
                            g->rlz ? size_t(5) * nv * n_r * n_lam * bk * 8 : 0, mats.size() * 8};
    size_t off[10] = {0};
    for (int i = 0; i < 9; i++) off[i + 1] = off[i] + ((need[i] + 255) & ~size_t(255));
    RegBlock ws(g, off[9]);
    if (ws.e != cudaSuccess) {
        set_error("regular grid buffers: %s", cudaGetErrorString(ws.e));
        return ws.e == cudaErrorMemoryAllocation ? SS_OUT_OF_MEMORY : SS_CUDA_ERROR;
    }
    char *at = (char *)ws.p;
    double *d_coef = (double *)(at + off[0]), *d_w = (double *)(at + off[1]), *d_tc = (double *)(at + off[3]);
    double *d_ts = (double *)(at + off[4]), *d_sr = (double *)(at + off[5]), *d_out = (double *)(at + off[6]);
    double *d_fb = (double *)(at + off[7]), *d_mats = (double *)(at + off[8]);
    int *d_m0 = (int *)(at + off[2]);
    auto run = [&]() -> int32_t {
        CUDA_TRY(cudaMemcpyAsync(d_w, w.data(), w.size() * 8, cudaMemcpyHostToDevice, st));
        CUDA_TRY(cudaMemcpyAsync(d_m0, m0.data(), m0.size() * 4, cudaMemcpyHostToDevice, st));
        if (dev_tables) {
            double *d_lam = d_tc + size_t(K) * n_lam;
            CUDA_TRY(cudaMemcpyAsync(d_lam, lam_pts, size_t(n_lam) * 8, cudaMemcpyHostToDevice, st));
            const int64_t ne = int64_t(K) * n_lam;
            if (ne > 0) reg_table_kernel<<<(unsigned)((ne + 127) / 128), 128, 0, st>>>(d_lam, d_tc, d_ts, K, n_lam);
            CUDA_TRY(cudaGetLastError());
        } else {
            CUDA_TRY(cudaMemcpyAsync(d_tc, tc.data(), tc.size() * 8, cudaMemcpyHostToDevice, st));
            CUDA_TRY(cudaMemcpyAsync(d_ts, ts.data(), ts.size() * 8, cudaMemcpyHostToDevice, st));
        }
        if (g->rlz) CUDA_TRY(cudaMemcpyAsync(d_mats, mats.data(), mats.size() * 8, cudaMemcpyHostToDevice, st));
        // SAtransform! of every slot
        int nmax = 0;
        for (auto &sh : g->spl_host) nmax = std::max(nmax, sh.Min);
        const int ld = (b % 2) ? b : b + 1;
        int optin = 0;
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, g->device);
        int per = 32;
        auto sa_smem = [&](int p) { return (size_t(p) * ld + size_t(5) * nmax) * 8; };
        while (per > 1 && sa_smem(per) > (size_t)optin) per /= 2;
        if (sa_smem(per) > (size_t)optin) {
            set_error("regularGridTransform: %d radial coefficients exceed shared memory", b);
            return SS_BAD_SHAPE;
        }
        CUDA_TRY(cudaFuncSetAttribute(reg_sa_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sa_smem(per)));
        reg_sa_kernel<P><<<dim3((ns + per - 1) / per, nitems), per, sa_smem(per), st>>>(
            (const P *)g->spec, g->d_spl, d_coef, d.n_spectral, b, ld, ns, bk);
        CUDA_TRY(cudaGetLastError());
        reg_si_kernel<<<dim3((ns + 127) / 128, n_r, nitems), 128, 0, st>>>(d_coef, d_m0, d_w, d_sr, b, ns, n_r,
                                                                            nitems);
        CUDA_TRY(cudaGetLastError());
        const size_t fsm = size_t(3) * ns * 8;  // the bound of an earlier kernel that staged whole rows: kept for callers
        if (fsm > (size_t)optin) {
            set_error("regularGridTransform: %d wavenumber slots exceed shared memory", ns);
            return SS_BAD_SHAPE;
        }
        reg_fourier_kernel<<<dim3((n_lam + 127) / 128, n_r, nitems), 128, 0, st>>>(
            d_sr, d_tc, d_ts, g->rlz ? d_fb : d_out, ns, K, n_r, n_lam, nitems, g->rlz, bk, nv);
        CUDA_TRY(cudaGetLastError());
        if (g->rlz) {
            const size_t msm = size_t(3) * n_z * bk * 8;
            if (msm > (size_t)optin) {
                set_error("regularGridTransform: %d z points exceed shared memory", n_z);
                return SS_BAD_SHAPE;
            }
            CUDA_TRY(cudaFuncSetAttribute(reg_cheb_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msm));
            const int64_t ncol = int64_t(n_r) * n_lam;
            const int64_t blocks = std::min<int64_t>((ncol * n_z + 255) / 256, 4096);
            reg_cheb_kernel<<<dim3((unsigned)blocks, nv, 5), 256, msm, st>>>(d_fb, d_mats, d_out, ncol, n_z, bk,
                                                                             nv, n_r);
            CUDA_TRY(cudaGetLastError());
        }
        // While the kernels run, map the result's pages (a fresh array has none): the copy
        // engine's own page faults take 2.4 ms of the 62 MB result of 61 × 361 × 25 points
        // and 2 variables, the copy into mapped pages 0.36 ms.
        const size_t page = (size_t)std::max<long>(sysconf(_SC_PAGESIZE), 4096) / 8;
        for (size_t i = 0; i < out_elems; i += page) ((volatile double *)out_host)[i] = 0.0;
        CUDA_TRY(cudaMemcpyAsync(out_host, d_out, out_elems * 8, cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaStreamSynchronize(st));
        return SS_OK;
    };
    const int32_t rc = run();
    if (rc) cudaStreamSynchronize(st);
    return rc ? rc : digit_status(g);
}

// Spline coefficients of every spectral block of `src` (FP64, [item][slot][b]) into a
// fresh device buffer (the caller frees it)
template <typename P>
int32_t block_coefficients(ss_grid *src, double **d_coef, cudaStream_t st) {
    const ss_dims &d = src->d;
    const int b = (int)d.b_iDim, ns = src->nslots_z, bk = (int)d.b_kDim;
    int nmax = 0;
    for (auto &sh : src->spl_host) nmax = std::max(nmax, sh.Min);
    const int ld = (b % 2) ? b : b + 1;
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, src->device);
    int per = 32;
    auto sa_smem = [&](int q) { return (size_t(q) * ld + size_t(5) * nmax) * 8; };
    while (per > 1 && sa_smem(per) > (size_t)optin) per /= 2;
    if (sa_smem(per) > (size_t)optin) {
        set_error("%d radial coefficients exceed shared memory", b);
        return SS_BAD_SHAPE;
    }
    CUDA_TRY(cudaMalloc(d_coef, size_t(src->nitems) * ns * b * 8));
    CUDA_TRY(cudaFuncSetAttribute(reg_sa_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sa_smem(per)));
    reg_sa_kernel<P><<<dim3((ns + per - 1) / per, src->nitems), per, sa_smem(per), st>>>(
        (const P *)src->spec, src->d_spl, *d_coef, d.n_spectral, b, ld, ns, bk);
    CUDA_TRY(cudaGetLastError());
    return SS_OK;
}

// The point kernel over host-described points: radii r (SI windows built here),
// angles, optional z, modes and taper weights; `out` is device memory
int32_t eval_points(ss_grid *g, const double *coef, const std::vector<double> &r, const std::vector<double> &lam,
                    const std::vector<double> &z, const std::vector<int> &mode, const std::vector<double> &taper,
                    const std::vector<double> &zcol, void *out, int64_t ostride_v, int out_f32, cudaStream_t st) {
    const ss_dims &d = g->d;
    const int64_t npts = (int64_t)r.size();
    if (npts == 0) return SS_OK;
    std::vector<int> m0;
    std::vector<double> w3;
    spline_point_weights(g->spl_host[0], r.data(), (int)npts, m0, w3);  // every variable shares the knots
    std::vector<double> w(size_t(npts) * 4);
    std::copy(w3.begin(), w3.begin() + w.size(), w.begin());  // d = 0: the value weights
    std::vector<double> ca;
    const int N = (int)d.kDim, bk = (int)d.b_kDim, nv = (int)d.nvars;
    if (g->rlz) {
        ca.assign(size_t(nv) * N * bk, 0.0);
        for (int v = 0; v < nv; v++) {
            ChebHost ch;
            int32_t rc = build_cheb(N, bk, g->bcb[v], g->bct[v], g->p.kMin, g->p.kMax, ch);
            if (rc) return rc;
            for (int n = 0; n < N; n++)  // CA[n][i] = δ_ni + Σ_p v_p[n] u_p[i]
                for (int i = 0; i < bk; i++) {
                    double a = (n == i) ? 1.0 : 0.0;
                    for (int q = 0; q < ch.nrank; q++) a += ch.gv[size_t(q) * N + n] * ch.gu[size_t(q) * bk + i];
                    ca[(size_t(v) * N + n) * bk + i] = a;
                }
        }
    }
    std::vector<void *> bufs;
    auto up = [&](const void *h, size_t bytes, void **dptr) -> cudaError_t {
        if (!bytes) { *dptr = nullptr; return cudaSuccess; }
        cudaError_t e = cudaMalloc(dptr, bytes);
        if (e != cudaSuccess) return e;
        bufs.push_back(*dptr);
        return cudaMemcpyAsync(*dptr, h, bytes, cudaMemcpyHostToDevice, st);
    };
    PointArgs A{};
    cudaError_t e = cudaSuccess;
    void *p_lam, *p_z, *p_w, *p_t, *p_m0, *p_mode, *p_ca, *p_zc;
    if ((e = up(lam.data(), lam.size() * 8, &p_lam)) || (e = up(z.data(), z.size() * 8, &p_z)) ||
        (e = up(w.data(), w.size() * 8, &p_w)) || (e = up(taper.data(), taper.size() * 8, &p_t)) ||
        (e = up(m0.data(), m0.size() * 4, &p_m0)) || (e = up(mode.data(), mode.size() * 4, &p_mode)) ||
        (e = up(ca.data(), ca.size() * 8, &p_ca)) || (e = up(zcol.data(), zcol.size() * 8, &p_zc))) {
        cudaStreamSynchronize(st);
        for (void *q : bufs) cudaFree(q);
        set_error("point evaluation buffers: %s", cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? SS_OUT_OF_MEMORY : SS_CUDA_ERROR;
    }
    A.coef = coef; A.lam = (const double *)p_lam; A.z = (const double *)p_z; A.w = (const double *)p_w;
    A.taper = (const double *)p_t; A.m0 = (const int *)p_m0; A.mode = (const int *)p_mode;
    A.ca = (const double *)p_ca; A.zcol = (const double *)p_zc; A.out = out;
    A.npts = npts; A.ostride_v = ostride_v; A.b = (int)d.b_iDim; A.nslots = g->nslots_z; A.K = (int)d.kDim_wn;
    A.bk = bk; A.nvars = nv; A.N = N; A.n_z = (int)zcol.size(); A.rlz = g->rlz; A.out_f32 = out_f32;
    A.zmin = g->p.kMin; A.zmax = g->p.kMax; A.first_var = 0; A.nvar_eval = nv;
    const int64_t warps = npts * nv;
    point_eval_kernel<<<(unsigned)((warps + 3) / 4), 128, size_t(4) * bk * 8, st>>>(A);
    e = cudaGetLastError();
    cudaError_t e2 = cudaStreamSynchronize(st);
    for (void *q : bufs) cudaFree(q);
    if (e != cudaSuccess || e2 != cudaSuccess) {
        set_error("point evaluation: %s", cudaGetErrorString(e != cudaSuccess ? e : e2));
        return SS_CUDA_ERROR;
    }
    return SS_OK;
}

template <typename P>
int32_t unstructured(ss_grid *g, const double *pts, int64_t npts, double *out, int oob, double fill,
                     cudaStream_t st) {
    const double rmin = g->p.iMin, rmax = g->p.iMax, zmin = g->p.kMin, zmax = g->p.kMax;
    std::vector<double> r(npts), lam(npts), z(g->rlz ? npts : 0), taper;
    std::vector<int> mode(npts, 0);
    int64_t n_oob = 0;
    for (int64_t i = 0; i < npts; i++) {
        r[i] = pts[i];
        lam[i] = pts[npts + i];
        bool in = r[i] >= rmin && r[i] <= rmax;  // _check_bounds_nd: Fourier λ is always in bounds
        if (g->rlz) {
            z[i] = pts[2 * npts + i];
            in = in && z[i] >= zmin && z[i] <= zmax;
        }
        if (!in) {
            mode[i] = 2;
            r[i] = std::min(std::max(r[i], rmin), rmax);
            n_oob++;
        }
    }
    if (oob == 1 && n_oob) {
        set_error("%lld points are outside the source domain", (long long)n_oob);
        return SS_BAD_ARG;
    }
    const int nv = (int)g->d.nvars;
    double *d_coef = nullptr, *d_out = nullptr;
    int32_t rc = block_coefficients<P>(g, &d_coef, st);
    if (rc) return rc;
    if (cudaMalloc((void **)&d_out, size_t(npts) * nv * 8) != cudaSuccess) {
        cudaGetLastError();
        cudaStreamSynchronize(st);
        cudaFree(d_coef);
        set_error("out of device memory");
        return SS_OUT_OF_MEMORY;
    }
    rc = eval_points(g, d_coef, r, lam, z, mode, taper, {}, d_out, npts, 0, st);
    if (!rc && cudaMemcpy(out, d_out, size_t(npts) * nv * 8, cudaMemcpyDeviceToHost) != cudaSuccess) {
        set_error("point evaluation download: %s", cudaGetErrorString(cudaGetLastError()));
        rc = SS_CUDA_ERROR;
    }
    cudaFree(d_coef);
    cudaFree(d_out);
    if (!rc && oob == 2)
        for (int64_t i = 0; i < npts; i++)
            if (mode[i] == 2)
                for (int v = 0; v < nv; v++) out[size_t(v) * npts + i] = fill;
    return rc ? rc : digit_status(g);
}

// relocate_grid / relocate_grid! fast path (src/relocation.jl:144-439): every
// gridpoint of the target evaluates the source at its shifted position
template <typename P>
int32_t relocate(ss_grid *t, ss_grid *s, double dx, double dy, int boundary, int taper_width, cudaStream_t st) {
    const ss_dims &d = s->d;
    const double rmin = s->p.iMin, rmax = s->p.iMax;
    const double DX = (rmax - rmin) / s->p.num_cells;
    const double r_start = taper_width > 0 ? rmax - taper_width * DX : rmax;
    const int64_t nring_pts = d.jDim;
    std::vector<double> r(nring_pts), lam(nring_pts), taper(nring_pts, 1.0), zcol;
    std::vector<int> mode(nring_pts, 0);
    const double twopi = 2 * 3.14159265358979323846;
    int64_t q = 0;
    for (int ri0 = 0; ri0 < (int)d.iDim; ri0++) {
        const int ri = ri0 + 1 + s->pOL, L = 4 + 4 * ri;
        const double ymin = 0.5 * (twopi / L) * (ri - 1), rm = s->spl_host[0].mish[ri0];
        for (int l = 0; l < L; l++, q++) {
            const double ln = ymin + twopi * l / L;
            const double xo = rm * std::cos(ln) + dx, yo = rm * std::sin(ln) + dy;
            const double ro = std::sqrt(xo * xo + yo * yo);
            lam[q] = std::atan2(yo, xo);
            const bool oob = ro > rmax || ro < rmin;
            r[q] = oob ? std::min(std::max(ro, rmin + 1e-10), rmax - 1e-10) : ro;
            if (oob) mode[q] = boundary == 0 ? 2 : (boundary == 2 ? 1 : 0);  // nan / nearest / azimuthal mean
            else if (taper_width > 0 && r[q] > r_start)
                taper[q] = 0.5 * (1.0 + std::cos(3.14159265358979323846 * (r[q] - r_start) / (rmax - r_start)));
        }
    }
    if (s->rlz) {
        ChebHost ch;
        int32_t rc = build_cheb((int)d.kDim, (int)d.b_kDim, s->bcb[0], s->bct[0], s->p.kMin, s->p.kMax, ch);
        if (rc) return rc;
        zcol = ch.mish;  // the column's Chebyshev points, zmin → zmax
    }
    double *d_coef = nullptr;
    int32_t rc = block_coefficients<P>(s, &d_coef, st);
    if (rc) return rc;
    rc = eval_points(s, d_coef, r, lam, {}, mode, taper, zcol, t->phys, d.n_physical, t->esz == 4, st);
    cudaFree(d_coef);
    if (rc) return rc;
    if ((rc = grid_forward(t, st))) return rc;  // spectralTransform!(target); gridTransform!(target)
    return grid_inverse(t, st);
}

}  // namespace

extern "C" int32_t ss_regular_grid_transform(ss_grid *g, const double *r_pts, int32_t n_r, const double *lam_pts,
                                             int32_t n_lam, const double *z_pts, int32_t n_z, double *out,
                                             void *stream) {
    if (!g || !r_pts || !lam_pts || !out || n_r < 1 || n_lam < 1) {
        set_error("regularGridTransform: null pointer or empty point set");
        return SS_BAD_ARG;
    }
    if (g->rlz && (!z_pts || n_z < 1)) {
        set_error("regularGridTransform: RLZ grids need z points");
        return SS_BAD_ARG;
    }
    CUDA_TRY(cudaSetDevice(g->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : g->stream;
    if (g->esz == 4) return regular<float>(g, r_pts, n_r, lam_pts, n_lam, z_pts, n_z, out, st);
    return regular<double>(g, r_pts, n_r, lam_pts, n_lam, z_pts, n_z, out, st);
}

extern "C" int32_t ss_evaluate_unstructured(ss_grid *g, const double *pts, int64_t npts, double *out,
                                            int32_t out_of_bounds, double fill, void *stream) {
    if (!g || !pts || !out || npts < 0 || out_of_bounds < 0 || out_of_bounds > 2) {
        set_error("evaluate_unstructured: bad arguments");
        return SS_BAD_ARG;
    }
    if (npts == 0) return SS_OK;
    CUDA_TRY(cudaSetDevice(g->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : g->stream;
    if (g->esz == 4) return unstructured<float>(g, pts, npts, out, out_of_bounds, fill, st);
    return unstructured<double>(g, pts, npts, out, out_of_bounds, fill, st);
}

extern "C" int32_t ss_relocate_grid(ss_grid *target, ss_grid *source, double dx, double dy, int32_t boundary,
                                    int32_t taper_width, void *stream) {
    if (!target || !source || boundary < 0 || boundary > 2 || taper_width < 0) {
        set_error("relocate_grid: bad arguments");
        return SS_BAD_ARG;
    }
    if (target->rlz != source->rlz || target->d.n_physical != source->d.n_physical ||
        target->d.nvars != source->d.nvars || target->esz != source->esz || target->device != source->device ||
        target->d.n_spectral != source->d.n_spectral) {
        set_error("relocate_grid: target must be a grid with the source's parameters");
        return SS_BAD_SHAPE;
    }
    CUDA_TRY(cudaSetDevice(source->device));
    // queued on the target's stream (where the caller's later work on the target
    // goes), after the source's queued work has finished
    cudaStream_t st = stream ? (cudaStream_t)stream : target->stream;
    CUDA_TRY(cudaStreamSynchronize(source->stream));
    if (const int32_t rc = digit_status(source)) return rc;
    if (source->esz == 4) return relocate<float>(target, source, dx, dy, boundary, taper_width, st);
    return relocate<double>(target, source, dx, dy, boundary, taper_width, st);
}
