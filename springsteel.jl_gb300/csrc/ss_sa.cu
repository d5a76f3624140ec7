// ss_sa.cu — SAtransform! + SI of binary64 and binary32 grids (no periodic
// spline): a banded LDLᵀ solve of 32 spectral slots per CTA in shared memory.
//
// SAtransform! (src/CubicBSpline.jl:1368-1396) solves Γ(P+Q)Γᵀ x = Γ(b − PQ·ahat)
// per slot and unfolds a = Γᵀ x + ahat; SI / SIx / SIxx evaluate 4-tap windows of a
// at the mish points.  An FP64 operation of a warp holds its scheduler's FP64 unit
// for 64 cycles here, whatever the active lanes, so what counts is the FP64
// operations per row and that the solving warps of an SM sit on different
// schedulers.  The factor is kept as unit-lower M and D (M = L·diag(L)^-1): 3 FMAs
// forward and 4 operations backward per row, one FMA on the dependent chain.
//
// Binary32 grids solve in binary64 as well and round x once: the value a binary32 solve
// with an FP64 refinement step (15 FP64 operations and ten conversions a row) is after, at
// any scale and along the whole slot (60-bit fixed point took 1.4 ms less on the 400-cell
// grid and as long elsewhere, but held a slot at one exponent; widening and rounding by
// integer operations took 0.8 ms more than the conversions).
//
// Measured before → here: 400-cell, 64-level binary32 RLZ grid of 4 variables 10.0 → 8.1 ms,
// 251-cell binary32 RL grid of 4 variables 0.88 → 0.15 ms, 125-cell, 40-level binary32 RLZ
// grid of 2 variables 0.59 → 0.19 ms, 200-cell FP64 RLZ grid of 5 variables 2.03 → 1.39 ms (12
// FP64 operations per slot and ring for SI alone hold the FP64 units for 0.85 ms),
// 100-cell FP64 RL grid 0.13 → 0.05 ms (a chain of 103 rows × 7 × 64 cycles).
#include <cuda_runtime.h>

#include <algorithm>

#include "ss_kernels.h"
#include "ss_types.cuh"

namespace ss {

constexpr int kSaWarps = 8;  // one solves, all load and evaluate
constexpr int kSaLd = 33;  // slots of a CTA + 1: rows of a slot and slots of a row are both conflict-free

// One warp solves its 32 slots in place; x: the lane's interior rows, row i at [i * kSaLd].
// Lane j holds row base + j of the factor, the next 32 rows already loading; a row's
// entries are broadcast by shuffles, off the dependent chain.
__device__ __forceinline__ void solve_f64(const SplineDev &sp, double *xi, int n, int lane, bool mine) {
    const double2 *ldl = reinterpret_cast<const double2 *>(sp.ldl);  // row i: (m1, m2), (m3, 1/d)
    auto factor = [&](int row, double2 &f0, double2 &f1) {
        const int r = min(max(row, 0), n - 1);
        f0 = __ldg(ldl + 2 * r);
        f1 = __ldg(ldl + 2 * r + 1);
    };
    double2 f0, f1, g0, g1;
    factor(lane, f0, f1);
    // forward: z_i = part_i − m1_{i−1} z_{i−1}, part_{i+1} = x_{i+1} − m3_{i−2} z_{i−2} − m2_{i−1} z_{i−1}
    double z0 = 0.0, z1 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0, m3b = 0.0;  // z_{i−1}, z_{i−2}; the columns'
    double part = xi[0];
    for (int base = 0; base < n; base += 32) {
        factor(base + 32 + lane, g0, g1);
        const int rows = min(32, n - base);
#pragma unroll 8
        for (int j = 0; j < rows; j++) {
            const int i = base + j;
            const double xn = xi[min(i + 1, n - 1) * kSaLd];
            const double z = part - m1 * z0;
            part = xn - m3b * z1;
            part -= m2 * z0;
            if (mine) xi[i * kSaLd] = z;
            z1 = z0; z0 = z;
            m1 = __shfl_sync(0xffffffffu, f0.x, j);
            m2 = __shfl_sync(0xffffffffu, f0.y, j);
            m3b = m3;
            m3 = __shfl_sync(0xffffffffu, f1.x, j);
        }
        f0 = g0; f1 = g1;
    }
    __syncwarp();
    // backward: x_i = part_i − m1_i x_{i+1}, part_{i−1} = z_{i−1}/d_{i−1} − m3_{i−1} x_{i+2} − m2_{i−1} x_{i+1}
    const int top = (n - 1) / 32 * 32;
    factor(top + lane, f0, f1);
    double x1 = 0.0, x2 = 0.0;  // x_{i+1}, x_{i+2}
    part = xi[(n - 1) * kSaLd] * __shfl_sync(0xffffffffu, f1.y, (n - 1) & 31);
    for (int base = top; base >= 0; base -= 32) {
        factor(base - 32 + lane, g0, g1);
#pragma unroll 8
        for (int j = min(32, n - base) - 1; j >= 0; j--) {
            const int i = base + j;
            const int jp = (j + 31) & 31;  // row i − 1: this batch, or the last of the next
            const double zp = xi[max(i - 1, 0) * kSaLd];
            const double n2 = __shfl_sync(0xffffffffu, j ? f0.y : g0.y, jp), n3 = __shfl_sync(0xffffffffu, j ? f1.x : g1.x, jp);
            const double nd = __shfl_sync(0xffffffffu, j ? f1.y : g1.y, jp), n1 = __shfl_sync(0xffffffffu, f0.x, j);
            const double xv = part - n1 * x1;
            part = zp * nd;
            part -= n3 * x2;
            part -= n2 * x1;
            if (mine) xi[i * kSaLd] = xv;
            x2 = x1; x1 = xv;
        }
        f0 = g0; f1 = g1;
    }
}

template <typename P, typename T>
__device__ __forceinline__ void sa_band_body(const SaLaunch &A, const int bx, const int by, const int part, const int parts) {
    static_assert(std::is_same<P, T>::value, "storage and compute types agree");
    constexpr bool kF32 = std::is_same<T, float>::value;
    extern __shared__ __align__(16) unsigned char sa_raw[];
    double *X = reinterpret_cast<double *>(sa_raw);  // [row][slot]; a float (before and after the solve) lies in the low word
    const int item = by;
    const int v = item / A.bk, zb = item % A.bk;
    const SplineDev &sp = A.spl[v];
    const int b = A.b, n = sp.Min, rL = sp.rankL;
    const int s0 = bx * 32, nsl = min(32, A.nslots_z - s0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const P *spec = (const P *)A.spec + (size_t)v * A.nspec + ((size_t)zb * A.nslots_z + s0) * b;
    for (int sl = warp; sl < nsl; sl += kSaWarps)
        for (int i = lane; i < b; i += 32) cp_async<sizeof(P)>(&X[i * kSaLd + sl], spec + (size_t)sl * b + i);
    cp_async_wait_all();
    __syncthreads();
    auto coef = [&](int i, int sl) -> T & { return *reinterpret_cast<T *>(&X[i * kSaLd + sl]); };

    if (!A.coeffs) {
        if constexpr (kF32) {
            for (int sl = warp; sl < nsl; sl += kSaWarps)
                for (int i = lane; i < b; i += 32) X[i * kSaLd + sl] = (double)coef(i, sl);
            __syncthreads();
        }
        const double *ah0 = (sp.r3x && A.ahat) ? A.ahat + ((size_t)v * A.nblocks + (size_t)zb * A.nslots_z + s0) * b : nullptr;
        if (ah0) {  // b̃ = b − PQ·ahat (full P+Q, half-width 3)
            for (int sl = warp; sl < nsl; sl += kSaWarps) {
                const double *ah = ah0 + (size_t)sl * b;
                for (int i = lane; i < b; i += 32) {
                    double acc = 0.0;
                    for (int j = max(0, i - 3); j <= min(b - 1, i + 3); j++) acc += sp.PQb[i * 7 + (j - i + 3)] * ah[j];
                    X[i * kSaLd + sl] -= acc;
                }
            }
            __syncthreads();
        }
        // CTAs of an SM solve on different schedulers
        if (warp == (bx & 3)) {
            double *x = X + min(lane, nsl - 1), *xi = x + rL * kSaLd;
            // the boundary terms of the Γ fold (src/CubicBSpline.jl:427-463)
            if (lane < nsl) {
                const double b0 = x[0], b1 = x[kSaLd], bM1 = x[(b - 1) * kSaLd], bM2 = x[(b - 2) * kSaLd];
                if (sp.lk == BC_A1) {
                    xi[0] += sp.aL * b0;
                    xi[kSaLd] += sp.bL * b0;
                } else if (sp.lk == BC_A2) {
                    xi[0] += sp.aL * b0 + sp.bL * b1;
                }
                if (sp.rk == BC_A1) {
                    xi[(n - 1) * kSaLd] += sp.aR * bM1;
                    xi[(n - 2) * kSaLd] += sp.bR * bM1;
                } else if (sp.rk == BC_A2) {
                    xi[(n - 1) * kSaLd] += sp.aR * bM1 + sp.bR * bM2;
                }
            }
            __syncwarp();
            solve_f64(sp, xi, n, lane, lane < nsl);
        }
        __syncthreads();
        // the solution in the compute type; Γᵀ x (src/CubicBSpline.jl:465-500) and the background
        for (int sl = warp; sl < nsl; sl += kSaWarps) {
            const double *ah = ah0 ? ah0 + (size_t)sl * b : nullptr;
            auto sol = [&](int i) -> T {  // interior row i, rounded
                return (T)X[(rL + i) * kSaLd + sl];
            };
            const T x0 = sol(0), x1 = sol(1), xn1 = sol(n - 1), xn2 = sol(n - 2);
            __syncwarp();
            for (int i = lane; i < b; i += 32) {
                T a = T(0);
                if (i >= rL && i < rL + n) a = sol(i - rL);
                else if (i < rL) {
                    if (sp.lk == BC_A1) a = i == 0 ? (T)sp.aL * x0 + (T)sp.bL * x1 : T(0);
                    if (sp.lk == BC_A2) a = i == 0 ? (T)sp.aL * x0 : (i == 1 ? (T)sp.bL * x0 : T(0));
                } else {
                    if (sp.rk == BC_A1) a = i == b - 1 ? (T)sp.aR * xn1 + (T)sp.bR * xn2 : T(0);
                    if (sp.rk == BC_A2) a = i == b - 1 ? (T)sp.aR * xn1 : (i == b - 2 ? (T)sp.bR * xn1 : T(0));
                }
                coef(i, sl) = ah ? (T)((double)a + ah[i]) : a;
            }
        }
        __syncthreads();
    }

    // f, ∂r, ∂rr at the mish points of the rings that carry the slots (s < 1 + 2ri),
    // four rings of a warp at a time so that their tables' loads overlap
    const int s = s0 + lane;
    const int first = max(0, (s0 - 1) / 2 - A.pOL);
    T *G = (T *)A.G + (size_t)item * A.frows + s;
    const size_t plane = (size_t)A.nitems * A.frows;
    const int slot = min(lane, nsl - 1);
    for (int r0 = first + (part * kSaWarps + warp) * 4; r0 < A.iDim; r0 += parts * kSaWarps * 4) {
        int m0[4];
        int64_t fo[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int r = min(r0 + q, A.iDim - 1);
            m0[q] = __ldg(sp.si_m0 + r);
            fo[q] = __ldg(A.fofs + r);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int r = min(r0 + q, A.iDim - 1);
            const bool live = r0 + q < A.iDim && lane < nsl && s < 1 + 2 * (r + 1 + A.pOL);
            const T a0 = coef(m0[q], slot), a1 = coef(m0[q] + 1, slot), a2 = coef(m0[q] + 2, slot), a3 = coef(m0[q] + 3, slot);
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const int64_t w = ((int64_t)d * A.iDim + r) * 4;
                const T u = ld_real<T>(sp.siw_t, w) * a0 + ld_real<T>(sp.siw_t, w + 1) * a1 +
                            ld_real<T>(sp.siw_t, w + 2) * a2 + ld_real<T>(sp.siw_t, w + 3) * a3;
                if (live) G[d * plane + fo[q]] = u;
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kSaWarps * 32) sa_band_kernel(SaLaunch A) {
    sa_band_body<T, T>(A, blockIdx.x, blockIdx.y, blockIdx.z, gridDim.z);
}
// fused multi-grid launch: CTA blockIdx.x runs work[blockIdx.x] (bz: part << 8 | parts); the record is
// staged in shared memory
template <typename T>
__global__ void __launch_bounds__(kSaWarps * 32) sa_band_fused_kernel(const SaLaunch *recs, const BatchWork *work) {
    __shared__ __align__(16) SaLaunch A;
    const BatchWork w = work[blockIdx.x];
    for (int i = threadIdx.x; i < (int)(sizeof(SaLaunch) / 4); i += blockDim.x)
        reinterpret_cast<int *>(&A)[i] = __ldg(reinterpret_cast<const int *>(recs + w.rec) + i);
    __syncthreads();
    sa_band_body<T, T>(A, w.bx, w.by, w.bz >> 8, w.bz & 255);
}

size_t sa_band_smem(int b) { return (size_t)b * kSaLd * sizeof(double); }

template <typename T>
cudaError_t launch_sa_band(const SaLaunch &A, int nitems, int sms, cudaStream_t st) {
    const size_t smem = sa_band_smem(A.b);
    // the process's attribute: one value for all grids, so that launches of other threads never lower it
    const cudaError_t e = cudaFuncSetAttribute(sa_band_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSaBandSmemMax);
    if (e != cudaSuccess) return e;
    // few CTAs: every one solves its slots again for a part of the rings only, so that
    // the evaluation (12 FP64 operations per slot and ring) spreads over idle SMs
    const int ctas = (A.nslots_z + 31) / 32 * nitems;
    const int parts = std::max(1, std::min({8, 2 * sms / ctas, (A.iDim + 31) / 32}));
    sa_band_kernel<T><<<dim3((A.nslots_z + 31) / 32, nitems, parts), kSaWarps * 32, smem, st>>>(A);
    return cudaGetLastError();
}
template <typename T>
cudaError_t launch_sa_band_fused(const SaLaunch *recs, const BatchWork *work, int nwork, size_t smem, cudaStream_t st) {
    if (nwork <= 0) return cudaSuccess;
    const cudaError_t e =
        cudaFuncSetAttribute(sa_band_fused_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSaBandSmemMax);
    if (e != cudaSuccess) return e;
    sa_band_fused_kernel<T><<<nwork, kSaWarps * 32, smem, st>>>(recs, work);
    return cudaGetLastError();
}
template cudaError_t launch_sa_band<double>(const SaLaunch &, int, int, cudaStream_t);
template cudaError_t launch_sa_band<float>(const SaLaunch &, int, int, cudaStream_t);
template cudaError_t launch_sa_band_fused<double>(const SaLaunch *, const BatchWork *, int, size_t, cudaStream_t);
template cudaError_t launch_sa_band_fused<float>(const SaLaunch *, const BatchWork *, int, size_t, cudaStream_t);

}  // namespace ss
