// ss_digit.cu — the ring DFTs of FP64 grids (binary32 RLZ grids: four inverse outputs)
// on the tensor cores, by products of digit slices.
//
// A ring of L = 4n points carries the wavenumbers k ≤ n − 1 only, and its points
// are symmetric about 0 and π/2, so HC2R of a column folds into four real
// products of quadrant size (cos / sin × even / odd k, n × n/2 each).  One ring
// holds nvars · b_kDim · 5 columns, so each product is a GEMM of the ring's own
// cosine matrix with the columns of all items.  FP64 runs at 2 FMA per clock and
// SM on this GPU and the mixed-radix FFT of the arbitrary lengths 4 + 4ri spends
// 2.3 times the conventional operations on prime factors; a binary16 tensor-core
// product with binary32 accumulation is exact while the operands are integers
// and the sums stay below 2^24 (see below).  So each column is scaled by the exponent of its
// largest entry to a fixed-point number and cut into balanced digits (Ozaki et
// al. 2012, error-free splitting), the matrix likewise once per grid, and
//     Σ_k Y[m][k] X[k][c] = Σ_s 2^{−9s} D_s,   D_s = Σ_{i+j=s} Σ_k y_i x_j,
// keeps s ≤ 6 (binary64; 26 of the 36 products, the rest is below 2^−60 of the
// column's scale) or s ≤ 2 (binary32).  The D_s are combined as integers in
// 64-bit fixed point (binary64) or in binary32.
//
// The sums are drained after at most 96 products.  Random digits then make them 2^19 (rms).
// Data whose digits follow the signs of a matrix row's could take D_3, D_4, D_5 and D_6 to 1.15,
// 1.30, 1.54 and 1.03 times 2^24 (computed from the cosine digits, n = 930; up to n = 193, drains of
// 64 products, every sum stays below): such a sum loses its last bit, 2^-44, 2^-53, 2^-62 and
// 2^-71 of the scale of one term.  Draining after 48 products excludes it for every n and costs
// 12 % of both directions of the 200-cell grid (inverse 12.7 → 14.3 ms).
//
// The reference turns each coefficient by cos, sin of the Float64 product k·ymin;
// the folded matrices hold the exact angles, and the difference δ_k (up to 1e-13)
// is applied to the fixed-point coefficients, so both agree to their last bits.
//
// Measured on the 200-cell, 32-level, 5-variable FP64 grid: ring_inverse 34.1 →
// 5.3 ms and ring_forward 7.1 → 1.9 ms, each with an error against 64-bit ring sums
// no larger than the FFT kernels' (9.2e-16 against 9.6e-16 of f, 3.0e-16 against
// 3.3e-16 of the spectral array at 200 cells).
//
// Binary32 RLZ grids take the four derivative outputs this way (f keeps the FFT's
// rounding, which a later ∂rr amplifies by r's spline, and so does the forward
// direction): 400 cells, 64 levels, 4 variables ring_inverse 29.9 → 17.6 ms.
//
// digit_split   G (spectra at the mish points) → column exponents and digit
//               planes in the MMA operand layout
// digit_gemm    persistent, warp-specialised: bulk copies → 8-slot (6-slot) ring
//               of K-steps → two issuing warps, one per accumulator half → sixteen
//               warps drain and combine both
// digit_unfold  quadrant parts → ring points (RL, and columns too long for the kernels that
//               read the parts)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <iterator>
#include <map>
#include <memory>
#include <mutex>
#include <utility>

#include "ss_digit.h"
#include "ss_digit_dev.cuh"
#include "ss_grid.h"
#include "ss_internal.h"
#include "ss_kernels.h"
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

namespace ss {

// ------------------------------------------------------------ tables
// cos(2πt/8n)·2^53, t = 0..2n, of every ring
__global__ void digit_cos_kernel(const DigitRing *rings, long long *cosq) {
    const DigitRing r = rings[blockIdx.x];
    const double inv = 1.0 / (4.0 * r.n);
    for (int t = threadIdx.x; t <= 2 * r.n; t += blockDim.x)
        cosq[r.cosofs + t] = __double2ll_rn((t <= r.n ? cospi(t * inv) : sinpi((2 * r.n - t) * inv)) * 0x1p53);
}
__device__ __forceinline__ long long quarter_cos(const long long *c, int n, int t) {  // 0 ≤ t < 8n
    if (t > 4 * n) t = 8 * n - t;
    return t > 2 * n ? -c[4 * n - t] : c[t];
}
// entry of part `part` at row m, wavenumber k, times 2^53 (`half`: half weight at k = 0,
// the inverse's result is doubled)
__device__ __forceinline__ long long dft_entry(const DigitRing &r, const long long *c, int part, int m, int k, bool half) {
    if (k > r.kmax || m >= r.n + 1 - r.half) return 0;
    const int per = 8 * r.n;
    int t = (int)((long long)k * (2 * m + r.half) % per);
    if (part >= 2) {  // −sin = −cos(t − 2n)
        t = t - 2 * r.n;
        if (t < 0) t += per;
        return -quarter_cos(c, r.n, t);
    }
    const long long v = quarter_cos(c, r.n, t);
    return half && k == 0 ? v / 2 : v;
}

// digit planes of the inverse matrices: A tile = [digit][row group][K core][8 rows][8 k]
// (forward: rows are wavenumbers and K the quadrant positions, without the half weight)
template <typename T, bool kForward>
__global__ void __launch_bounds__(256) digit_matrix_kernel(const DigitRing *rings, const long long *cosq, uint8_t *A) {
    const DigitRing r = rings[blockIdx.x];
    const long long *c = cosq + r.cosofs;
    const int64_t ntile = kForward ? (int64_t)4 * r.rtf * r.tm : (int64_t)r.rt * 2 * (r.te + r.to);
    for (int64_t e = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; e < ntile * 256; e += (int64_t)gridDim.y * blockDim.x) {
        const int64_t tile = e >> 8;
        const int row = (int)(e & 127), kg = (int)((e >> 7) & 1);
        int part = 0;
        int64_t q = tile;
        int steps = r.tm;
        if (kForward) {
            part = (int)(tile / (r.rtf * r.tm));
            q = tile - (int64_t)part * r.rtf * r.tm;
        } else {
            while (part < 3 && tile >= digit_part_base(r, part + 1, r.rt)) part++;
            steps = digit_steps(r, part);
            q = tile - digit_part_base(r, part, r.rt);
        }
        const int m = (int)(q / steps) * kDigitRows + row, j0 = (int)(q % steps) * 16 + kg * 8;
        auto entry = [&](int i) {
            if (!kForward) return dft_entry(r, c, part, m, 2 * (j0 + i) + (part & 1), true);
            return dft_entry(r, c, part, j0 + i, 2 * m + (part & 1), false);
        };
        uint8_t *dst = A + ((kForward ? r.af_tile : r.a_tile) + tile) * digit_a_bytes<T>() + (row >> 3) * 256 + kg * 128 + (row & 7) * 16;
        if constexpr (std::is_same<T, double>::value) {
            unsigned long long U[8];
#pragma unroll
            for (int i = 0; i < 8; i++) U[i] = kDigitBias + (unsigned long long)entry(i);
            uint4 w[6];
            planes8<true>(U, w);
#pragma unroll
            for (int i = 0; i < 6; i++) *reinterpret_cast<uint4 *>(dst + i * kDigitPlane) = w[i];
        } else {
            // 28-bit fixed point, rounded from the 53 bits: a leading digit and two of base 1024
            uint32_t w[3][4];
#pragma unroll
            for (int q2 = 0; q2 < 4; q2++) {
                float d[3][2];
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const int X = (int)((entry(2 * q2 + p) + (1 << 24)) >> 25);
                    const int d2 = ((X + 512) & 1023) - 512, X1 = (X - d2) >> 10;
                    const int d1 = ((X1 + 512) & 1023) - 512;
                    d[2][p] = (float)d2;
                    d[1][p] = (float)d1;
                    d[0][p] = (float)((X1 - d1) >> 10);
                }
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const __half2 h = __floats2half2_rn(d[i][0], d[i][1]);
                    w[i][q2] = *reinterpret_cast<const uint32_t *>(&h);
                }
            }
#pragma unroll
            for (int i = 0; i < 3; i++)
                *reinterpret_cast<uint4 *>(dst + i * kDigitPlane) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
        }
    }
}

// ------------------------------------------------------------ split
// CTA = (ring of the span, group of 8 items).  Pass 1: a warp per item finds the
// largest exponent of each variant's column (k·X and k²·X for ∂λ, ∂λλ); pass 2:
// a thread per (item, source, 16 wavenumbers), source = real or imaginary parts
// of even or odd k, writes 8 K entries of each plane as 16 bytes; the 8 items of
// a group are the 8 rows of one core matrix, so a warp's stores are 128-byte
// runs.  Column of (item, variant): (item / 8)·8·kVars + variant·8 + item mod 8.
// Joined: the items of many RL grids with the same rings are the items of one product.
// They are ordered by falling ring count, so ring r holds the first count[r] of them.
struct DigitItemRef {
    const double *in, *G;      // slot 1 and G of the item
    double *F, *out;           // F; slot 1
    long long *H;              // quadrant parts
    int64_t gplane, hplane, oplane;  // to the next derivative of G, output of H, slot
    int *err;
    int cap;
};
struct DigitJoin {
    const DigitItemRef *refs;
    const int *count;
};

struct SplitArgs {
    const void *G;
    const DigitRing *rings;
    const int64_t *btile;
    uint8_t *B;
    int *expo;
    const int *delta, *cap;   // cap: largest wavenumber of every item (per-variable kmax of RL grids)
    int64_t frows;
    int r0, nitems, iDim, col_tiles;
    DigitJoin join;
};
template <typename T>
SS_HD constexpr int inverse_col_tiles(int items) {
    return ((items + kDigitGroup - 1) / kDigitGroup * kDigitGroup * DigitFormat<T>::kVars + 2 * DigitFormat<T>::kCols - 1) /
           (2 * DigitFormat<T>::kCols);
}
SS_HD constexpr int forward_col_tiles(int items) {
    return (items + 2 * DigitFormat<double>::kCols - 1) / (2 * DigitFormat<double>::kCols);
}

__device__ __forceinline__ uint32_t mag_bits(double v) { return (uint32_t)__double2hiint(v) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t mag_bits(float v) { return (uint32_t)__float_as_int(v) & 0x7fffffffu; }
template <typename T>
__device__ __forceinline__ int mag_expo(uint32_t bits) {  // biased exponent ≥ 1, or kNanColumn
    if constexpr (std::is_same<T, double>::value) {
        const int e = (int)(bits >> 20);
        return e == 0x7ff ? kNanColumn : (e > 0 ? e : 1);
    } else {
        const int e = (int)(bits >> 23);
        return e == 0xff ? kNanColumn : (e > 0 ? e : 1);
    }
}

template <typename T, bool kJoin>
__global__ void __launch_bounds__(256, 2) digit_split_kernel(SplitArgs S) {
    using F = DigitFormat<T>;
    constexpr int V0 = kDigitVariants - F::kVars;
    __shared__ int ex[kDigitGroup][kDigitVariants];
    const int ring = S.r0 + (int)(gridDim.y - 1 - blockIdx.y);  // largest rings first
    const DigitRing r = S.rings[ring];
    const int grp = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int here = kJoin ? S.join.count[ring] : S.nitems;  // items of this ring
    if (kJoin && grp * kDigitGroup >= here) return;
    auto row_of = [&](int item, size_t &plane, int &cap) {
        if constexpr (kJoin) {
            const DigitItemRef &q = S.join.refs[item];
            plane = (size_t)q.gplane;
            cap = q.cap;
            return (const T *)q.G + r.fofs;
        } else {
            plane = (size_t)S.nitems * S.frows;
            cap = S.cap[item];
            return (const T *)S.G + (size_t)item * S.frows + r.fofs;
        }
    };
    {
        const int item = grp * kDigitGroup + warp;
        uint32_t mx[kDigitVariants] = {0, 0, 0, 0, 0};
        if (item < here) {
            size_t plane;
            int cap;
            const T *g0 = row_of(item, plane, cap);
            const int kmax = min(r.kmax, cap);
            for (int s = lane; s < 1 + 2 * kmax; s += 32) {
                const T k = (T)((s + 1) >> 1);
                const T v = g0[s];
                mx[0] = max(mx[0], mag_bits(v));
                mx[1] = max(mx[1], mag_bits(v * k));
                mx[2] = max(mx[2], mag_bits(v * k * k));
                mx[3] = max(mx[3], mag_bits(g0[s + plane]));
                mx[4] = max(mx[4], mag_bits(g0[s + 2 * plane]));
            }
        }
#pragma unroll
        for (int q = 0; q < kDigitVariants; q++) {
            const int e = mag_expo<T>(__reduce_max_sync(0xffffffffu, mx[q]));
            if (lane == 0) {
                ex[warp][q] = e;
                // of the parts: one higher where the products store them halved
                const int up = std::is_same<T, double>::value && r.n > kDigitFullRing && e != kNanColumn ? 1 : 0;
                if (item < here) S.expo[((size_t)q * S.nitems + item) * S.iDim + ring] = e + up;
            }
        }
    }
    __syncthreads();
    // warp-uniform control flow: lanes exchange values; idle ones (no such item, no
    // such odd step) read item 0 and store nothing
    const int il = threadIdx.x & 7;
    const bool real = grp * kDigitGroup + il < here;
    const int item = real ? grp * kDigitGroup + il : 0;
    const int par = (threadIdx.x >> 3) & 1, imag = (threadIdx.x >> 4) & 1;
    const int64_t bt = S.btile[ring];
    size_t plane;
    int cap;
    const T *g = row_of(item, plane, cap);
    const int kmax = min(r.kmax, cap);
    const int steps = par ? r.to : r.te;
    const int col_tiles = kJoin ? inverse_col_tiles<T>(here) : S.col_tiles;
    for (int kg = warp; kg < 2 * r.te; kg += 8) {
        const bool store = real && kg < 2 * steps;
        const int k0 = 16 * kg + par;
        int dk[8];
        if constexpr (std::is_same<T, double>::value) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int k = k0 + 2 * i;
                dk[i] = (k > 0 && k <= kmax) ? S.delta[r.dofs + k - 1] : 0;
            }
        }
#pragma unroll 1
        for (int d = 0; d < 3; d++) {
            T x[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int k = k0 + 2 * i;
                x[i] = (k <= kmax && (k > 0 || !imag)) ? g[d * plane + (k > 0 ? 2 * k - 1 + imag : 0)] : T(0);
            }
#pragma unroll 1
            for (int dl = 0; dl < (d == 0 ? 3 : 1); dl++) {
                if (dl > 0) {  // ×ik: (re, im) → (−k im, k re)
                    const bool neg = (dl == 1) == (imag != 0);
#pragma unroll
                    for (int i = 0; i < 8; i++) x[i] *= (T)(neg ? -(k0 + 2 * i) : k0 + 2 * i);
                }
                const int var = d == 0 ? dl : d + 2;
                if (var < V0) continue;
                const int part = ((imag ^ (dl & 1)) << 1) + par;
                const int e = ex[il][var];
                const int col = (grp * F::kVars + var - V0) * kDigitGroup + il;
                const int ct = col / (2 * F::kCols), cl = col % (2 * F::kCols);
                const int h = cl / F::kCols, c = cl % F::kCols;
                uint4 w[F::kDigits];
                if constexpr (std::is_same<T, double>::value) {
                    // cos entries −= δ·sin entries, sin += δ·cos: the partner lane holds the
                    // other half of the same wavenumbers
                    unsigned long long U[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const long long X = fixed_point<54>(x[i], e);
                        const int other = __shfl_xor_sync(0xffffffffu, (int)(X >> 23), 16);
                        const int turn = (__mulhi(other, dk[i]) + (1 << 14)) >> 15;
                        U[i] = kDigitBias + (unsigned long long)(part < 2 ? X - turn : X + turn);
                    }
                    planes8(U, w);
                } else {
                    float y[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) y[i] = scale2(x[i], 8 - (e - 126));
                    planes8(y, w);
                }
                const int64_t tile = bt + digit_part_base(r, part, col_tiles) + (int64_t)ct * steps + (kg >> 1);
                uint8_t *dst = S.B + tile * digit_b_bytes<T>() + h * digit_half_bytes<T>() + (kg & 1) * 128 + (c & 7) * 16;
                if (store)
#pragma unroll
                    for (int i = 0; i < F::kDigits; i++)
                        *reinterpret_cast<uint4 *>(dst + ((i * F::kCols + c) >> 3) * 256) = w[i];
            }
        }
    }
}

// ------------------------------------------------------------ product
struct GemmDigitArgs {
    const uint8_t *A, *B;
    const DigitItem *items;
    int nwork;
    const DigitRing *rings;
    const int *expo;
    void *out;
    int64_t jDim, frows;
    int nitems, nvars, bk, iDim;
    int *err;
    DigitJoin join;
};

constexpr int kDrainWarps = 16;
constexpr int kDigitThreads = (kDrainWarps + 3) * 32;  // and 1 copying, 2 issuing warps

// One CTA per SM (shared-memory ring, 2 × kSums·kCols accumulator columns).
// Each accumulator half has its own issuing warp, so one half computes while the
// sixteen draining warps, which serve both, are at the other.
template <typename T, bool kForward, bool kJoin>
__global__ void __launch_bounds__(kDigitThreads, 1) digit_gemm_kernel(GemmDigitArgs g) {
    using F = DigitFormat<T>;
    constexpr int ND = F::kDigits, W = F::kCols, ST = F::kStages;
    constexpr uint32_t AB = digit_a_bytes<T>(), HB = digit_half_bytes<T>(), BB = digit_b_bytes<T>();
    extern __shared__ __align__(1024) uint8_t dsm[];
    __shared__ __align__(8) uint64_t full[ST], empty[ST], accf[2], acce[2], drain[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int quit;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < ST; i++) {
            bar_init(&full[i], 1);
            bar_init(&empty[i], 2);
        }
        for (int h = 0; h < 2; h++) {
            bar_init(&accf[h], 1);
            bar_init(&acce[h], kDrainWarps * 32);
            bar_init(&drain[h], 1);
        }
        quit = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (warp == kDrainWarps) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            DigitItem next = g.items[blockIdx.x];
            for (int w = blockIdx.x; ok && w < g.nwork; w += gridDim.x) {
                const DigitItem d = next;
                if (w + gridDim.x < g.nwork) next = g.items[w + gridDim.x];
                const uint8_t *a = g.A + d.a_tile * AB, *b = g.B + d.b_tile * BB;
                for (int k = 0; k < d.steps; k++, it++) {
                    const uint32_t s = it % ST;
                    if (!(ok = bar_wait(&empty[s], ((it / ST) & 1) ^ 1, &quit))) break;
                    const uint32_t dst = smem_addr(dsm + s * (AB + BB)), bar = smem_addr(&full[s]);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(AB + BB) : "memory");
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                                 "l"(a + (size_t)k * AB), "r"(AB), "r"(bar)
                                 : "memory");
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst + AB),
                                 "l"(b + (size_t)k * BB), "r"(BB), "r"(bar)
                                 : "memory");
                }
            }
            if (!ok) {  // copies in flight land before the CTA leaves
                int never = 0;
                for (uint32_t q = it > ST ? it - ST : 0; q < it; q++) bar_wait(&full[q % ST], (q / ST) & 1, &never);
            }
        }
    } else if (warp > kDrainWarps) {
        if (lane == 0) {
            const int h = warp - kDrainWarps - 1;
            const uint32_t tacc = tmem + h * 256;
            uint32_t it = 0, ch = 0;
            bool ok = true;
            int next = g.items[blockIdx.x].steps;
            for (int w = blockIdx.x; ok && w < g.nwork; w += gridDim.x) {
                const int steps = next;
                if (w + gridDim.x < g.nwork) next = g.items[w + gridDim.x].steps;
                const int nch = (steps + F::kChunk - 1) / F::kChunk, len = (steps + nch - 1) / nch;
                for (int k0 = 0; ok && k0 < steps; k0 += len, ch++) {
                    if (!(ok = bar_wait(&acce[h], (ch & 1) ^ 1, &quit))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const int ke = min(len, steps - k0);
                    for (int k = 0; k < ke; k++, it++) {
                        const uint32_t s = it % ST;
                        if (!(ok = bar_wait(&full[s], (it / ST) & 1, &quit))) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t sa = smem_addr(dsm + s * (AB + BB));
                        const uint64_t bd = operand_desc(sa + AB + h * HB);
                        if constexpr (F::kSums > ND) {
                            // digit i of the matrix times the data digits j ≤ kSums − 1 − i; the
                            // first step writes D_1..D_6 by i = 1, then D_0, then adds the rest of i = 0
                            static_assert(F::kSums == ND + 1, "D_6 is the only sum without a digit-0 term");
                            const bool first = k == 0;
                            if (first) {
                                mma_f16(tacc + W, operand_desc(sa + kDigitPlane), bd, mma_idesc(ND * W), 0u);
                                mma_f16(tacc, operand_desc(sa), bd, mma_idesc(W), 0u);
                                mma_f16(tacc + W, operand_desc(sa), operand_desc(sa + AB + h * HB + W * 32), mma_idesc((ND - 1) * W), 1u);
                            } else {
                                mma_f16(tacc, operand_desc(sa), bd, mma_idesc(ND * W), 1u);
                                mma_f16(tacc + W, operand_desc(sa + kDigitPlane), bd, mma_idesc(ND * W), 1u);
                            }
#pragma unroll
                            for (int i = 2; i < ND; i++)
                                mma_f16(tacc + i * W, operand_desc(sa + i * kDigitPlane), bd, mma_idesc((F::kSums - i) * W), 1u);
                        } else {
#pragma unroll
                            for (int i = 0; i < ND; i++)
                                mma_f16(tacc + i * W, operand_desc(sa + i * kDigitPlane), bd, mma_idesc((ND - i) * W),
                                        (k > 0 || i > 0) ? 1u : 0u);
                        }
                        mma_commit(&empty[s]);
                    }
                    mma_commit(&accf[h]);
                }
            }
            if (!ok) {
                int never = 0;
                mma_commit(&drain[h]);
                bar_wait(&drain[h], 0, &never);
            }
        }
    } else {
        // every draining warp owns 32 rows and a quarter of each half's columns, so a
        // half is drained by all of them in turn and is soon free for its issuer
        constexpr int WC = W / 4;
        const int cb = (warp >> 2) * WC;
        const uint32_t tacc = tmem + ((uint32_t)((warp & 3) * 32) << 16) + cb;
        uint32_t ch = 0;
        bool ok = true;
        for (int w = blockIdx.x; ok && w < g.nwork; w += gridDim.x) {
            const DigitItem d = g.items[w];
            const int nch = (d.steps + F::kChunk - 1) / F::kChunk;
            const DigitRing *r = g.rings + d.ring;
            const int row = d.row_tile * kDigitRows + (warp & 3) * 32 + lane;
            // forward rows: wavenumber k = 2·row + parity ≤ ri, stored at slot 2k − 1 (re), 2k (im)
            const int k = 2 * row + (d.part & 1);
            const int m = kForward ? max(2 * k - 1 + (d.part >> 1), 0) : row - r->lo[d.part];
            const bool live = kForward ? k < r->n && (k > 0 || d.part == 0) : m >= 0 && m < r->cnt[d.part];
            const int here = kJoin ? g.join.count[d.ring] : g.nitems;
            // lane c's column of this warp (half c / WC): its output row (null for padding) and exponent
            using Acc = typename std::conditional<std::is_same<T, double>::value, unsigned long long, float>::type;
            auto col_base = [&](int c, int &e) -> Acc * {
                constexpr int V0 = kDigitVariants - F::kVars;
                const int col = (d.col_tile * 2 + c / WC) * W + cb + c % WC;
                const int item = col / (kDigitGroup * F::kVars) * kDigitGroup + col % kDigitGroup;
                const int var = col / kDigitGroup % F::kVars + V0;
                e = 0;
                if constexpr (kForward) {
                    if (c >= 2 * WC || col >= here) return nullptr;
                    e = g.expo[(size_t)col * g.iDim + d.ring];
                    if constexpr (kJoin) return (Acc *)g.join.refs[col].F + r->fofs;
                    return (Acc *)g.out + (int64_t)col * g.frows + r->fofs;
                }
                if (c >= 2 * WC || item >= here) return nullptr;
                e = g.expo[((size_t)var * g.nitems + item) * g.iDim + d.ring];
                if constexpr (kJoin) return (Acc *)g.join.refs[item].H + var * g.join.refs[item].hplane + r->jofs + r->off[d.part];
                return (Acc *)g.out + ((int64_t)var * g.nvars + item / g.bk) * g.bk * g.jDim + (int64_t)g.bk * r->jofs + r->off[d.part] +
                       (int64_t)(item % g.bk) * r->L;
            };
            using Comb = Combine<false>;
            Acc V[2 * WC];
            const Acc start = std::is_same<T, double>::value ? (Acc)(0ull - Comb::kOffset * (unsigned)nch) : (Acc)0;
#pragma unroll
            for (int c = 0; c < 2 * WC; c++) V[c] = start;
            for (int q = 0; ok && q < nch; q++, ch++) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (!(ok = ok && __all_sync(0xffffffffu, bar_wait(&accf[h], ch & 1, &quit)))) continue;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int c0 = 0; c0 < WC; c0 += 4) {
                        float D[F::kSums][4];
#pragma unroll
                        for (int s = 0; s < F::kSums; s++) tmem_ld4(tacc + h * 256 + s * W + c0, D[s]);
                        tmem_wait_ld();
                        if (c0 + 4 == WC) {
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            bar_arrive(&acce[h]);
                        }
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            if constexpr (std::is_same<T, double>::value)
                                Comb::add(V[h * WC + c0 + c], D[0][c], D[1][c], D[2][c], D[3][c], D[4][c], D[5][c], D[6][c]);
                            else
                                V[h * WC + c0 + c] += fmaf(fmaf(D[2][c], 0x1p-10f, D[1][c]), 0x1p-10f, D[0][c]);
                        }
                    }
                }
            }
            if constexpr (!kForward && std::is_same<T, double>::value) {
                if (r->n > kDigitFullRing) {  // headroom for the four parts' sum
#pragma unroll
                    for (int c = 0; c < 2 * WC; c++) V[c] = (Acc)(((long long)V[c] + 1) >> 1);
                }
            }
            const double inv_len = kForward ? 1.0 / (double)r->L : 0.0;
#pragma unroll
            for (int c0 = 0; c0 < 2 * WC; c0 += 32) {
                int e;
                const long long mine = (long long)col_base(c0 + lane, e);
#pragma unroll
                for (int c = 0; c < 32; c++) {
                    if (c0 + c >= 2 * WC) break;
                    Acc *const base = (Acc *)__shfl_sync(0xffffffffu, mine, c);
                    Acc v = V[c0 + c];
                    if constexpr (std::is_same<T, float>::value) {
                        // doubled product of 2^-8 fixed-point operands at column scale 2^(e − 126)
                        const int ce = __shfl_sync(0xffffffffu, e, c);
                        v = ce == kNanColumn ? __int_as_float(0x7fc00000) : scale2(v, ce - 126 - 15);
                    }
                    if constexpr (kForward) {
                        // folded points scaled by 2^(e − 1020): Σ = V 2^(e − 1020 − 53)
                        const int ce = __shfl_sync(0xffffffffu, e, c);
                        if (ok && live && base)
                            ((double *)base)[m] = ce == kNanColumn ? __longlong_as_double(0x7ff8000000000000ll)
                                                                           : fixed_to_double((long long)v, ce + 1) * inv_len;
                    } else {
                        if (ok && live && base) base[m] = v;
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && quit) {
        if constexpr (kJoin)
            for (int i = 0; i < g.nitems; i++) *g.join.refs[i].err = 1;
        else *g.err = 1;
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ------------------------------------------------------------ unfold
// The four quadrant parts of one (ring, item, variant) row → its 4n points: in place
// (RLZ) or into the physical slot (RL, `phys` set)
struct UnfoldArgs {
    void *H, *phys;
    const DigitRing *rings;
    const int *expo;
    int64_t jDim;
    int r0, nitems, nvars, bk, iDim;
    DigitJoin join;
};
template <typename T, bool kJoin>
__global__ void __launch_bounds__(128) digit_unfold_kernel(UnfoldArgs U) {
    using R = typename std::conditional<std::is_same<T, double>::value, long long, float>::type;
    extern __shared__ __align__(16) unsigned char row_raw[];
    R *row = reinterpret_cast<R *>(row_raw);
    const int ring = U.r0 + (int)(gridDim.y - 1 - blockIdx.y), nitems = U.nitems;
    const DigitRing &r = U.rings[ring];
    const int n = r.n, L = r.L, shift = r.shift;
    const int var = blockIdx.x / nitems + kDigitVariants - DigitFormat<T>::kVars, item = blockIdx.x % nitems;
    const int slot = var == 0 ? 0 : (var < 3 ? var + 2 : var - 2);  // f, ∂r, ∂rr, ∂λ, ∂λλ
    const R *h;
    T *dst;
    if constexpr (kJoin) {
        if (item >= U.join.count[ring]) return;
        const DigitItemRef &q = U.join.refs[item];
        h = q.H + var * q.hplane + r.jofs;
        dst = q.out + slot * q.oplane + r.jofs;
    } else {
        const int64_t at = (int64_t)(item / U.bk) * U.bk * U.jDim + (int64_t)U.bk * r.jofs + (int64_t)(item % U.bk) * L;
        const int64_t out = (int64_t)var * U.nvars * U.bk * U.jDim + at;
        h = (const R *)U.H + out;
        dst = U.phys ? (T *)U.phys + (int64_t)slot * U.nvars * U.jDim + at : (T *)U.H + out;
    }
    for (int i = threadIdx.x; i < L; i += blockDim.x) row[i] = h[i];
    int e = 0;
    if constexpr (std::is_same<T, double>::value) e = U.expo[((size_t)var * nitems + item) * U.iDim + ring];
    __syncthreads();
    auto put = [&](int p, R v) {
        int l = p - shift;
        if (l < 0) l += L;
        if (l >= L) l -= L;
        if constexpr (std::is_same<T, double>::value)
            dst[l] = e == kNanColumn ? __longlong_as_double(0x7ff8000000000000ll) : fixed_to_double(v, e);
        else dst[l] = v;
    };
    for (int m = threadIdx.x; m < n; m += blockDim.x) {
        if (r.half == 0 && m == 0) {
            const R a = row[0], b = row[n + 1], c = row[n], d = row[3 * n + n - 1];
            put(0, a + b);
            put(2 * n, a - b);
            put(n, c + d);
            put(3 * n, c - d);
        } else {
            const R ce = row[m], co = row[r.off[1] + m], se = row[r.off[2] + m - r.lo[2]], so = row[r.off[3] + m - r.lo[3]];
            const R u = ce + co, v = ce - co, w = se + so, z = se - so;
            const int hf = r.half;
            put(m, u + w);
            put(4 * n - hf - m, u - w);
            put(2 * n - hf - m, v - z);
            put(2 * n + m, v + z);
        }
    }
}

// ------------------------------------------------------------ forward split and turn
// CTA = (ring of the span, group of 8 items).  Pass 1: a warp per item finds the
// largest exponent of its ring; pass 2: a thread per (item, cos or sin parts, 8
// quadrant positions) folds the four reflected points of each position in 62-bit
// fixed point (the folded parts are below 2^(expo − 1020)) and writes both parities.
struct FoldArgs {
    const double *C;
    const DigitRing *rings;
    const int64_t *btile;
    uint8_t *B;
    int *expo;
    int64_t jDim;
    int r0, nitems, iDim, bk, col_tiles;
    DigitJoin join;
};

template <bool kJoin>
__global__ void __launch_bounds__(256, 2) digit_fold_kernel(FoldArgs S) {
    using F = DigitFormat<double>;
    __shared__ int ex[kDigitGroup];
    const int ring = S.r0 + (int)(gridDim.y - 1 - blockIdx.y);
    const DigitRing r = S.rings[ring];
    const int grp = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int here = kJoin ? S.join.count[ring] : S.nitems;
    if (kJoin && grp * kDigitGroup >= here) return;
    auto row_of = [&](int item) {
        if constexpr (kJoin) return S.join.refs[item].in + r.jofs;
        return S.C + (int64_t)(item / S.bk) * S.bk * S.jDim + (int64_t)S.bk * r.jofs + (int64_t)(item % S.bk) * r.L;
    };
    {
        const int item = grp * kDigitGroup + warp;
        uint32_t mx = 0;
        if (item < here) {
            const double2 *x = reinterpret_cast<const double2 *>(row_of(item));  // even offsets and lengths
            for (int i = lane; i < r.L / 2; i += 32) {
                const double2 v = x[i];
                mx = max(mx, max(mag_bits(v.x), mag_bits(v.y)));
            }
        }
        const int e = mag_expo<double>(__reduce_max_sync(0xffffffffu, mx));
        if (lane == 0) {
            ex[warp] = e;
            if (item < here) S.expo[(size_t)item * S.iDim + ring] = e;
        }
    }
    __syncthreads();
    const int il = threadIdx.x & 7, item = grp * kDigitGroup + il;
    if (item >= here) return;
    const int col_tiles = kJoin ? forward_col_tiles(here) : S.col_tiles;
    const int sine = (threadIdx.x >> 3) & 1;
    const double *x = row_of(item);
    const int n = r.n, hf = r.half, L = r.L, e = ex[il];
    const int ct = item / (2 * F::kCols), cl = item % (2 * F::kCols), h = cl / F::kCols, c = cl % F::kCols;
    const int64_t bt = S.btile[ring] + (int64_t)ct * r.tm;
    for (int mg = threadIdx.x >> 4; mg < 2 * r.tm; mg += 16) {
        unsigned long long even[8], odd[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int m = mg * 8 + i;
            long long s = 0, d = 0;
            if (m < n + 1 - hf) {
                auto at = [&](int p) {
                    int l = p - r.shift;
                    if (l < 0) l += L;
                    if (l >= L) l -= L;
                    return fixed_point<60>(x[l], e);
                };
                // the axis positions hold two points, not four: m = 0 (θ = 0, π), m = n (θ = ±π/2)
                const bool axis0 = hf == 0 && m == 0, axis1 = hf == 0 && m == n;
                const long long a = at(m), b = axis0 ? 0 : at(4 * n - hf - m);
                const long long f = axis1 ? 0 : at(2 * n - hf - m), g = (axis0 || axis1) ? 0 : at(2 * n + m);
                s = sine ? a - b : a + b;
                d = sine ? f - g : f + g;
            }
            // cos: even s + d, odd s − d; sin: even s − d, odd s + d; 62 → 54 bits
            const long long u = s + d, w = s - d;
            even[i] = kDigitBias + (unsigned long long)(((sine ? w : u) + 128) >> 8);
            odd[i] = kDigitBias + (unsigned long long)(((sine ? u : w) + 128) >> 8);
        }
        uint4 w[6];
        const int64_t tile = bt + (int64_t)(2 * sine) * col_tiles * r.tm + (mg >> 1);
        uint8_t *dst = S.B + tile * digit_b_bytes<double>() + h * digit_half_bytes<double>() + (mg & 1) * 128 + (c & 7) * 16;
        planes8(even, w);
#pragma unroll
        for (int i = 0; i < 6; i++) *reinterpret_cast<uint4 *>(dst + ((i * F::kCols + c) >> 3) * 256) = w[i];
        dst += (int64_t)col_tiles * r.tm * digit_b_bytes<double>();
        planes8(odd, w);
#pragma unroll
        for (int i = 0; i < 6; i++) *reinterpret_cast<uint4 *>(dst + ((i * F::kCols + c) >> 3) * 256) = w[i];
    }
}

// X_k ← X_k e^{−iδ_k}: the forward coefficients at the reference's rounded angles,
// zero above the item's own kmax
struct TurnArgs {
    double *F;
    const DigitRing *rings;
    const int *delta, *cap;
    int64_t frows;
    int r0;
    DigitJoin join;
};
template <bool kJoin>
__global__ void __launch_bounds__(128) digit_turn_kernel(TurnArgs U) {
    const int ring = U.r0 + blockIdx.y, item = blockIdx.x;
    const DigitRing &r = U.rings[ring];
    if (kJoin && item >= U.join.count[ring]) return;
    double *f = (kJoin ? U.join.refs[item].F : U.F + (int64_t)item * U.frows) + r.fofs;
    const int kmax = min(r.kmax, kJoin ? U.join.refs[item].cap : U.cap[item]);
    const int *delta = U.delta;
    for (int k = kmax + 1 + threadIdx.x; k <= r.kmax; k += blockDim.x) f[2 * k - 1] = f[2 * k] = 0.0;
    for (int k = 1 + threadIdx.x; k <= kmax; k += blockDim.x) {
        const double d = (double)delta[r.dofs + k - 1] * 0x1p-70;
        const double re = f[2 * k - 1], im = f[2 * k];
        f[2 * k - 1] = fma(d, im, re);
        f[2 * k] = fma(-d, re, im);
    }
}

// ------------------------------------------------------------ host
// Least items (variables × Chebyshev modes) of a grid the products serve: FP64 grids
// of 3 items already run ring_inverse 4.2× (6 cells), 11.7× (37) and 3.3× (200 cells)
// faster than the FFT kernels, so the line lies at one.
constexpr int kDigitMinItems = 1;
// Binary32 (RLZ, the four derivatives), inverse rings + columns, FFT ÷ digits.  Items:
// 8 0.97 (100 cells), 0.88 (200), 0.83 (340); 16 1.02, 1.11, 1.05; 24 1.18, 1.24, 1.19.
// Points: the FFT kernels hold small grids on the chip at once, 60 cells 0.94 (2.9 million),
// 1.02 (5.3), 1.15 (11); 80 cells 1.01 (5.1); 100 cells 1.16 (4.0).  Rings: below 60 cells
// the matrices' tiles are mostly padding, 37 cells 1.00 (81 items), 0.88 (172), 20 cells 0.75.
constexpr int kDigitMinItemsF32 = 16, kDigitMinRingsF32 = 180;
constexpr int64_t kDigitMinPointsF32 = 3500000;
// bound of a grid's matrix digits (both directions: 4.5 GB at 200 cells, growing with
// the cube of the ring count); larger grids keep the FFT kernels
constexpr size_t kDigitTableBytes = (size_t)16 << 30;
// Tables above this many bytes are built while they take at most a quarter of the device's free
// memory, so that grids created later find room
constexpr size_t kDigitAskBytes = (size_t)256 << 20;
// RL grids hold far less data than these matrices (0.7 GB at 100 cells): up to about
// 120 cells.  100 cells, one variable: ring_inverse 1.07 → 0.13 ms, ring_forward
// 0.26 → 0.13 ms; 24 cells: 0.32 → 0.03 and 0.095 → 0.03 ms
constexpr size_t kDigitTableBytesRl = (size_t)1 << 30;
// spectra digits of one span of rings; larger grids take several spans
constexpr int64_t kDigitScratchBytes = (int64_t)1 << 30;
template <typename T>
constexpr size_t digit_smem() { return (size_t)DigitFormat<T>::kStages * (digit_a_bytes<T>() + digit_b_bytes<T>()); }

// Timed-out-wait flags, host memory that the kernels write: mapping a page takes 0.11 ms and giving
// it back 0.17, a quarter of creating a small grid, so the grids of the process share pages; a
// page goes with its last flag.
namespace {
struct FlagPage {
    int *base;
    std::vector<char> used;
    int live;
};
constexpr int kFlags = 512;
// (not destroyed at exit: a grid may be closed after the library's static objects)
std::mutex &flag_mutex = *new std::mutex;
std::vector<FlagPage> &flag_pages = *new std::vector<FlagPage>;
}  // namespace
static int *take_flag() {
    std::lock_guard<std::mutex> lock(flag_mutex);
    auto page = std::find_if(flag_pages.begin(), flag_pages.end(), [](const FlagPage &p) { return p.live < kFlags; });
    if (page == flag_pages.end()) {
        int *base = nullptr;
        if (cudaHostAlloc((void **)&base, kFlags * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        flag_pages.push_back({base, std::vector<char>(kFlags, 0), 0});
        page = flag_pages.end() - 1;
    }
    const int i = (int)(std::find(page->used.begin(), page->used.end(), 0) - page->used.begin());
    page->used[i] = 1;
    page->live++;
    page->base[i] = 0;
    return page->base + i;
}
static void give_flag(int *flag) {
    std::lock_guard<std::mutex> lock(flag_mutex);
    for (size_t k = 0; k < flag_pages.size(); k++) {
        FlagPage &p = flag_pages[k];
        if (flag < p.base || flag >= p.base + kFlags) continue;
        p.used[flag - p.base] = 0;
        if (--p.live == 0) {
            cudaFreeHost(p.base);
            flag_pages.erase(flag_pages.begin() + k);
        }
        return;
    }
}

// The matrix digits depend on the ring lengths and wavenumbers alone: grids of the same rings on a device
// share them (4.5 GB for 200 cells, 0.7 for an RL grid of 100).  They go with the last such grid.
struct DigitTables {
    void *A = nullptr;
    ~DigitTables() {
        if (A) cudaFree(A);
    }
};
namespace {
std::mutex &table_mutex = *new std::mutex;
auto &tables = *new std::map<std::vector<int>, std::weak_ptr<DigitTables>>;
}  // namespace

// B tiles of a ring, and its tile products with the first B tile at `used`
static int64_t ring_tiles(const DigitRing &q, int tiles, bool fwd) { return (int64_t)tiles * (fwd ? 4 * q.tm : 2 * (q.te + q.to)); }
static void ring_items(const DigitRing &q, int ring, int tiles, bool fwd, int64_t used, std::vector<DigitItem> &items) {
    for (int part = 0; part < 4; part++)
        for (int ct = 0; ct < tiles; ct++)
            for (int rt = 0; rt < (fwd ? q.rtf : q.rt); rt++) {
                const int steps = fwd ? q.tm : digit_steps(q, part);
                DigitItem it{};
                if (fwd) {
                    it.a_tile = q.af_tile + ((int64_t)part * q.rtf + rt) * steps;
                    it.b_tile = used + ((int64_t)part * tiles + ct) * steps;
                } else {
                    it.a_tile = q.a_tile + digit_part_base(q, part, q.rt) + (int64_t)rt * steps;
                    it.b_tile = used + digit_part_base(q, part, tiles) + (int64_t)ct * steps;
                }
                it.ring = ring; it.part = part; it.row_tile = rt; it.col_tile = ct; it.steps = steps;
                items.push_back(it);
            }
}

template <typename T>
static int32_t build(ss_grid *g, const std::vector<RingDesc> &rd) {
    using F = DigitFormat<T>;
    DigitPlan &D = g->digit;
    const int nr = (int)g->d.iDim;
    std::vector<DigitRing> rings(nr);
    int64_t cosn = 0, atiles = 0, aftiles = 0, dn = 0;
    for (int i = 0; i < nr; i++) {
        DigitRing &r = rings[i];
        std::memset(&r, 0, sizeof r);
        r.n = rd[i].ri + 1;
        r.L = rd[i].L;
        r.half = r.n & 1;
        r.shift = r.half ? (r.n - 3) / 2 : (r.n - 2) / 2;
        r.kmax = rd[i].kmax;
        for (size_t s = 1; s < rd.size() / nr; s++) r.kmax = std::max(r.kmax, rd[s * nr + i].kmax);  // RL: a set per variable
        r.te = (r.kmax / 2 + 1 + 15) / 16;
        r.to = std::max(1, ((r.kmax + 1) / 2 + 15) / 16);
        const int rows = r.n + 1 - r.half;
        r.rt = (rows + kDigitRows - 1) / kDigitRows;
        const int n = r.n;
        if (r.half) {
            for (int q = 0; q < 4; q++) { r.cnt[q] = n; r.lo[q] = 0; r.off[q] = q * n; }
        } else {
            const int cnt[4] = {n + 1, n, n - 1, n}, lo[4] = {0, 0, 1, 1}, off[4] = {0, n + 1, 2 * n + 1, 3 * n};
            for (int q = 0; q < 4; q++) { r.cnt[q] = cnt[q]; r.lo[q] = lo[q]; r.off[q] = off[q]; }
        }
        r.jofs = rd[i].jofs;
        r.fofs = rd[i].fofs;
        r.cosofs = cosn;
        cosn += 2 * n + 1;
        r.a_tile = atiles;
        atiles += (int64_t)r.rt * 2 * (r.te + r.to);
        r.tm = (rows + 15) / 16;
        r.rtf = ((n + 1) / 2 + kDigitRows - 1) / kDigitRows;
        r.af_tile = aftiles;
        aftiles += (int64_t)4 * r.rtf * r.tm;
        r.dofs = dn;
        dn += rd[i].ri;
    }
    // δ_k = fl(k·ymin) − k·(exact ymin): the product's rounding (exact by fma) and k times ymin's own
    std::vector<int> delta(std::max<int64_t>(dn, 1), 0);
    for (int i = 0; i < nr; i++) {
        const int ri = rd[i].ri, L = rd[i].L;
        const double ymin = 0.5 * (2 * 3.14159265358979323846 / L) * (ri - 1);
        const long double exact = 3.14159265358979323846264338327950288L * (ri - 1) / L;
        const double dy = (double)((long double)ymin - exact);
        for (int k = 1; k <= ri; k++) {
            const double a = k * ymin;
            delta[rings[i].dofs + k - 1] = (int)std::lrint(std::ldexp(k * dy - std::fma((double)k, ymin, -a), 70));
        }
    }
    D.col_tiles = inverse_col_tiles<T>(g->nitems);
    D.col_tiles_fwd = forward_col_tiles(g->nitems);
    constexpr bool kBoth = std::is_same<T, double>::value;  // binary32 grids keep the forward FFT's rounding
    const size_t abytes = (size_t)atiles * digit_a_bytes<T>(), afbytes = kBoth ? (size_t)aftiles * digit_a_bytes<T>() : 0;
    if (abytes + afbytes > (g->rlz ? kDigitTableBytes : kDigitTableBytesRl)) return SS_OK;
    DigitBlock blk;
    const size_t mark = g->allocs.size();
    auto give_up = [&]() {  // the device has no room for the tables: the FFT kernels serve
        cudaGetLastError();
        if (D.err) give_flag(D.err);
        while (g->allocs.size() > mark) { cudaFree(g->allocs.back()); g->allocs.pop_back(); }
        D = DigitPlan{};
        return SS_OK;
    };
    // spans of rings, largest first, whose B digits fit the scratch
    int64_t btiles = 0;
    auto make_set = [&](int lo, int hi, bool fwd, DigitSet &set) {
        const int tiles = fwd ? D.col_tiles_fwd : D.col_tiles;
        std::vector<DigitItem> items;
        std::vector<int64_t> btile(nr, 0);
        int r = hi;
        while (r > lo) {
            DigitSpan sp{0, r, (int)items.size(), 0};
            int64_t used = 0;
            while (r > lo) {
                const DigitRing &q = rings[r - 1];
                const int64_t need = ring_tiles(q, tiles, fwd);
                if (used > 0 && (used + need) * digit_b_bytes<T>() > kDigitScratchBytes) break;
                r--;
                btile[r] = used;
                ring_items(q, r, tiles, fwd, used, items);
                used += need;
            }
            sp.r0 = r;
            sp.items = (int)items.size() - sp.item0;
            btiles = std::max(btiles, used);
            set.spans.push_back(sp);
        }
        blk.put(&set.items, items);
        blk.put(&set.btile, btile);
    };
    blk.put(&D.rings, rings);
    D.ring_host = rings;
    blk.put(&D.delta, delta);
    std::vector<int> cap(g->nitems);
    for (int i = 0; i < g->nitems; i++) {
        const int km = g->rlz ? g->ring_kmax : g->kmaxv[i];
        cap[i] = km >= 0 ? km : rd[nr - 1].ri;
    }
    blk.put(&D.cap, cap);
    D.cap_host = cap;
    make_set(0, nr, false, D.whole);
    if (kBoth) make_set(0, nr, true, D.whole_fwd);
    const size_t nchunk = g->chunk_r0.size() - 1;
    D.chunks.resize(nchunk);
    D.chunks_fwd.resize(nchunk);
    for (size_t c = 0; c < nchunk && nchunk > 1; c++) {
        make_set(g->chunk_r0[c], g->chunk_r0[c + 1], false, D.chunks[c]);
        if (kBoth) make_set(g->chunk_r0[c], g->chunk_r0[c + 1], true, D.chunks_fwd[c]);
    }
    if (g->tl == TL_F32 && cheb_inverse_takes_quads((int)g->d.kDim, (int)g->d.b_kDim)) {
        std::vector<int2> blocks;
        D.quads.first.assign(1, 0);
        for (int r = 0; r < nr; r++) {
            for (int m = 0; m < rings[r].n; m += 16) blocks.push_back(make_int2(r, m));
            D.quads.first.push_back((int)blocks.size());
        }
        blk.put(&D.quads.blocks, blocks);
    }
    blk.room((void **)&D.expo, (size_t)kDigitVariants * g->nitems * nr * sizeof(int));
    blk.room(&D.B, std::max((size_t)btiles * digit_b_bytes<T>(), (size_t)cosn * 8));
    // quadrant parts (RLZ grids keep them in the ring outputs' buffer)
    if (!g->rlz) blk.room(&D.H, (size_t)kDigitVariants * g->nitems * g->d.jDim * sizeof(T));
    if (!blk.build(g->allocs)) return give_up();
    if (nchunk == 1) {  // the only chunk is the grid
        D.chunks[0] = D.whole;
        D.chunks_fwd[0] = D.whole_fwd;
    }
    if (!(D.err = take_flag())) return give_up();
    std::vector<int> key{g->device, g->tl};
    for (const DigitRing &r : rings) {
        key.push_back(r.n);
        key.push_back(r.kmax);
    }
    std::lock_guard<std::mutex> lock(table_mutex);  // of two threads one builds, the other finds them complete
    for (auto it = tables.begin(); it != tables.end();) it = it->second.expired() ? tables.erase(it) : std::next(it);
    if (const auto found = tables.find(key); found != tables.end()) D.tables = found->second.lock();
    if (!D.tables) {
        size_t left = 0, total = 0;
        if (abytes + afbytes > kDigitAskBytes &&
            (cudaMemGetInfo(&left, &total) != cudaSuccess || abytes + afbytes > left / 4))
            return give_up();
        auto t = std::make_shared<DigitTables>();
        if (cudaMalloc(&t->A, abytes + afbytes) != cudaSuccess) { t->A = nullptr; return give_up(); }
        long long *cosq = (long long *)D.B;  // scratch until the first transform
        uint8_t *A = (uint8_t *)t->A;        // whole tiles: Af is aligned
        digit_cos_kernel<<<nr, 128, 0, g->stream>>>(D.rings, cosq);
        digit_matrix_kernel<T, false><<<dim3(nr, 8), 256, 0, g->stream>>>(D.rings, cosq, A);
        if constexpr (kBoth) digit_matrix_kernel<T, true><<<dim3(nr, 8), 256, 0, g->stream>>>(D.rings, cosq, A + abytes);
        CUDA_TRY(cudaGetLastError());
        CUDA_TRY(cudaStreamSynchronize(g->stream));
        D.tables = t;
        tables[key] = t;
    }
    D.A = D.tables->A;
    if (kBoth) D.Af = (uint8_t *)D.A + abytes;
    CUDA_TRY(cudaFuncSetAttribute(digit_gemm_kernel<T, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)digit_smem<T>()));
    if constexpr (kBoth)
        CUDA_TRY(cudaFuncSetAttribute(digit_gemm_kernel<T, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)digit_smem<T>()));
    D.on = true;
    return SS_OK;
}

int32_t digit_build(ss_grid *g, const std::vector<RingDesc> &rings) {
    if (g->tl == TL_DF64 || (g->tl == TL_F32 && !g->rlz)) return SS_OK;
    int least = g->tl == TL_F64 ? kDigitMinItems : kDigitMinItemsF32;
    if (const char *e = std::getenv("SS_RING_DIGITS")) {  // tuning override: the least item count, 0 for never
        least = std::atoi(e);
        if (least <= 0) return SS_OK;
    } else if (g->tl == TL_F32 && (g->d.iDim < kDigitMinRingsF32 || g->d.jDim * g->nitems < kDigitMinPointsF32)) {
        return SS_OK;
    }
    if (g->nitems < least) return SS_OK;
    if (rings[g->d.iDim - 1].ri + 1 > (g->tl == TL_F64 ? kDigitMaxRing : kDigitMaxRingF32)) return SS_OK;
    return g->tl == TL_F64 ? build<double>(g, rings) : build<float>(g, rings);
}

void digit_free(ss_grid *g) {
    if (g->digit.err) give_flag(g->digit.err);
    g->digit.err = nullptr;
    g->digit.tables.reset();
}

int32_t digit_status(ss_grid *g) {
    volatile int *err = g->digit.err;
    if (!err || !*err) return SS_OK;
    *err = 0;
    set_error("ring product: a bounded device wait gave up");
    return SS_DEVICE_TIMEOUT;
}

// the kernels' arguments for one span of rings
static SplitArgs split_args(const ss_grid *g, const DigitSet &set, const DigitSpan &sp) {
    const DigitPlan &D = g->digit;
    return {g->G, D.rings, set.btile, (uint8_t *)D.B, D.expo, D.delta, D.cap, g->frows, sp.r0, g->nitems, (int)g->d.iDim, D.col_tiles};
}
static FoldArgs fold_args(const ss_grid *g, const DigitSet &set, const DigitSpan &sp) {
    const DigitPlan &D = g->digit;
    return {(const double *)(g->rlz ? g->C : g->phys), D.rings, set.btile, (uint8_t *)D.B, D.expo, g->d.jDim, sp.r0, g->nitems,
            (int)g->d.iDim, (int)g->d.b_kDim, D.col_tiles_fwd};
}
static GemmDigitArgs gemm_args(const ss_grid *g, const DigitSet &set, const DigitSpan &sp, bool fwd) {
    const DigitPlan &D = g->digit;
    return {(const uint8_t *)(fwd ? D.Af : D.A), (const uint8_t *)D.B, set.items + sp.item0, sp.items, D.rings, D.expo,
            fwd ? g->F : (D.H ? D.H : g->H), g->d.jDim, g->frows, g->nitems, (int)g->d.nvars, (int)g->d.b_kDim, (int)g->d.iDim, D.err};
}
static UnfoldArgs unfold_args(const ss_grid *g, const DigitSpan &sp) {
    const DigitPlan &D = g->digit;
    return {D.H ? D.H : g->H, g->rlz ? nullptr : g->phys, D.rings, D.expo, g->d.jDim, sp.r0, g->nitems, (int)g->d.nvars,
            (int)g->d.b_kDim, (int)g->d.iDim};
}
static TurnArgs turn_args(const ss_grid *g, const DigitSpan &sp) {
    const DigitPlan &D = g->digit;
    return {(double *)g->F, D.rings, D.delta, D.cap, g->frows, sp.r0};
}
static int split_groups(const ss_grid *g) { return (g->nitems + kDigitGroup - 1) / kDigitGroup; }
template <typename T>
static size_t unfold_smem(const ss_grid *g, const DigitSpan &sp) { return (size_t)4 * (sp.r1 + g->pOL + 1) * sizeof(T); }

template <typename T>
static int32_t inverse(ss_grid *g, cudaStream_t st, const DigitSet &set, int *launches) {
    const DigitPlan &D = g->digit;
    for (const DigitSpan &sp : set.spans) {
        const int nr = sp.r1 - sp.r0;
        digit_split_kernel<T, false><<<dim3(split_groups(g), nr), 256, 0, st>>>(split_args(g, set, sp));
        digit_gemm_kernel<T, false, false><<<std::min(g->sms, sp.items), kDigitThreads, digit_smem<T>(), st>>>(
            gemm_args(g, set, sp, false));
        *launches += 2;
        CUDA_TRY(cudaGetLastError());
        if (D.columns.on || D.quads.blocks) continue;  // the column stage reads the parts
        digit_unfold_kernel<T, false><<<dim3(DigitFormat<T>::kVars * g->nitems, nr), 128, unfold_smem<T>(g, sp), st>>>(unfold_args(g, sp));
        CUDA_TRY(cudaGetLastError());
        *launches += 1;
    }
    return SS_OK;
}

int32_t digit_ring_forward(ss_grid *g, cudaStream_t st, int chunk, int *launches) {
    const DigitSet &set = chunk < 0 ? g->digit.whole_fwd : g->digit.chunks_fwd[chunk];
    for (const DigitSpan &sp : set.spans) {
        const int nr = sp.r1 - sp.r0;
        digit_fold_kernel<false><<<dim3(split_groups(g), nr), 256, 0, st>>>(fold_args(g, set, sp));
        digit_gemm_kernel<double, true, false><<<std::min(g->sms, sp.items), kDigitThreads, digit_smem<double>(), st>>>(
            gemm_args(g, set, sp, true));
        digit_turn_kernel<false><<<dim3(g->nitems, nr), 128, 0, st>>>(turn_args(g, sp));
        CUDA_TRY(cudaGetLastError());
        *launches += 3;
    }
    return SS_OK;
}

// ---- joined
bool digit_joins(const ss_grid *g) {
    return g->digit.on && !g->rlz && g->tl == TL_F64 && g->digit.whole.spans.size() == 1 && g->digit.whole_fwd.spans.size() == 1;
}

// Grids whose common rings have the same matrices: same offset, and wavenumbers up to the
// same cap wherever a ring reaches it
static bool same_rings(const ss_grid *a, const ss_grid *b) {
    const std::vector<DigitRing> &x = a->digit.ring_host, &y = b->digit.ring_host;
    for (size_t i = 0; i < std::min(x.size(), y.size()); i++)
        if (x[i].n != y[i].n || x[i].kmax != y[i].kmax) return false;
    return true;
}

int32_t digit_join_plan(std::vector<ss_grid *> gs, std::vector<void *> &mem, std::vector<DigitJoined> &out) {
    std::stable_sort(gs.begin(), gs.end(), [](const ss_grid *a, const ss_grid *b) { return a->d.iDim > b->d.iDim; });
    auto alloc = [&](void **p, size_t bytes) -> int32_t {
        CUDA_TRY(cudaMalloc(p, std::max<size_t>(bytes, 16)));
        mem.push_back(*p);
        return SS_OK;
    };
    auto put = [&](const auto &v, auto **dst) -> int32_t {
        void *p = nullptr;
        const int32_t rc = alloc(&p, v.size() * sizeof(v[0]));
        if (rc) return rc;
        *dst = (typename std::remove_reference<decltype(**dst)>::type *)p;
        CUDA_TRY(cudaMemcpy(p, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice));
        return SS_OK;
    };
    const int64_t most = kDigitScratchBytes / digit_b_bytes<double>();
    while (!gs.empty()) {
        const ss_grid *first = gs[0];  // most rings: its matrices serve the set
        const std::vector<DigitRing> &rings = first->digit.ring_host;
        const int nr = (int)rings.size();
        std::vector<int> count(nr, 0);
        auto tiles_of = [&](bool fwd) {
            int64_t n = 0;
            for (int r = 0; r < nr; r++) n += ring_tiles(rings[r], fwd ? forward_col_tiles(count[r]) : inverse_col_tiles<double>(count[r]), fwd);
            return n;
        };
        std::vector<DigitItemRef> refs;
        std::vector<ss_grid *> rest;
        for (ss_grid *g : gs) {
            for (int r = 0; r < g->d.iDim; r++) count[r] += g->nitems;
            if (!refs.empty() && (!same_rings(first, g) || std::max(tiles_of(false), tiles_of(true)) > most)) {
                for (int r = 0; r < g->d.iDim; r++) count[r] -= g->nitems;
                rest.push_back(g);
                continue;
            }
            for (int v = 0; v < g->nitems; v++)  // RL: items are variables
                refs.push_back({(const double *)g->phys + v * g->d.jDim, (const double *)g->G + v * g->frows,
                                (double *)g->F + v * g->frows, (double *)g->phys + v * g->d.jDim,
                                (long long *)g->digit.H + v * g->d.jDim, g->nitems * g->frows, g->d.nvars * g->d.jDim,
                                g->d.nvars * g->d.jDim, g->digit.err, g->digit.cap_host[v]});
        }
        DigitJoined J;
        const DigitItemRef *dref = nullptr;
        const int *dcount = nullptr;
        int32_t rc = put(refs, &dref);
        if (rc || (rc = put(count, &dcount))) return rc;
        void *B = nullptr, *expo = nullptr;
        if ((rc = alloc(&B, (size_t)std::max(tiles_of(false), tiles_of(true)) * digit_b_bytes<double>()))) return rc;
        if ((rc = alloc(&expo, (size_t)kDigitVariants * refs.size() * nr * sizeof(int)))) return rc;
        J.refs = dref; J.count = dcount; J.B = B; J.expo = (int *)expo;
        J.owner = first; J.items = (int)refs.size();
        for (int fwd = 0; fwd < 2; fwd++) {
            std::vector<DigitItem> items;
            std::vector<int64_t> btile(nr);
            int64_t used = 0;
            for (int r = nr - 1; r >= 0; r--) {  // longest products first: the CTAs take them in turn
                const int tiles = fwd ? forward_col_tiles(count[r]) : inverse_col_tiles<double>(count[r]);
                btile[r] = used;
                ring_items(rings[r], r, tiles, fwd, used, items);
                used += ring_tiles(rings[r], tiles, fwd);
            }
            if ((rc = put(items, &J.work[fwd])) || (rc = put(btile, &J.btile[fwd]))) return rc;
            J.nwork[fwd] = (int)items.size();
        }
        CUDA_TRY(cudaFuncSetAttribute(digit_gemm_kernel<double, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)digit_smem<double>()));
        CUDA_TRY(cudaFuncSetAttribute(digit_gemm_kernel<double, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)digit_smem<double>()));
        out.push_back(J);
        gs.swap(rest);
    }
    return SS_OK;
}

cudaError_t digit_join_launch(const DigitJoined &J, bool fwd, cudaStream_t st) {
    const ss_grid *g = J.owner;
    const DigitPlan &D = g->digit;
    const DigitJoin join{(const DigitItemRef *)J.refs, J.count};
    const int nr = (int)g->d.iDim, groups = (J.items + kDigitGroup - 1) / kDigitGroup;
    const GemmDigitArgs A{(const uint8_t *)(fwd ? D.Af : D.A), (const uint8_t *)J.B, J.work[fwd], J.nwork[fwd], D.rings, J.expo, nullptr,
                          0, 0, J.items, 0, 1, nr, D.err, join};
    const int ctas = std::min(g->sms, J.nwork[fwd]);
    if (fwd) {
        const FoldArgs S{nullptr, D.rings, J.btile[1], (uint8_t *)J.B, J.expo, 0, 0, J.items, nr, 1, 0, join};
        digit_fold_kernel<true><<<dim3(groups, nr), 256, 0, st>>>(S);
        digit_gemm_kernel<double, true, true><<<ctas, kDigitThreads, digit_smem<double>(), st>>>(A);
        digit_turn_kernel<true><<<dim3(J.items, nr), 128, 0, st>>>({nullptr, D.rings, D.delta, nullptr, 0, 0, join});
    } else {
        const SplitArgs S{nullptr, D.rings, J.btile[0], (uint8_t *)J.B, J.expo, D.delta, nullptr, 0, 0, J.items, nr, 0, join};
        digit_split_kernel<double, true><<<dim3(groups, nr), 256, 0, st>>>(S);
        digit_gemm_kernel<double, false, true><<<ctas, kDigitThreads, digit_smem<double>(), st>>>(A);
        const size_t row = (size_t)4 * D.ring_host.back().n * sizeof(double);
        digit_unfold_kernel<double, true><<<dim3(kDigitVariants * J.items, nr), 128, row, st>>>(
            {nullptr, nullptr, D.rings, J.expo, 0, 0, J.items, 0, 1, nr, join});
    }
    return cudaGetLastError();
}

int32_t digit_ring_inverse(ss_grid *g, cudaStream_t st, int chunk, int *launches) {
    const DigitSet &set = chunk < 0 ? g->digit.whole : g->digit.chunks[chunk];
    return g->tl == TL_F64 ? inverse<double>(g, st, set, launches) : inverse<float>(g, st, set, launches);
}

}  // namespace ss

extern "C" int32_t ss_grid_digits(const ss_grid *g, int32_t *stages) {
    if (!g || !stages) { set_error("null argument"); return SS_BAD_ARG; }
    const DigitPlan &D = g->digit;
    *stages = !D.on ? 0 : (g->tl == TL_F64 ? SS_DIGITS_RING_FWD : 0) | SS_DIGITS_RING_INV |
                              (D.columns.fon ? SS_DIGITS_CHEB_FWD : 0) | (D.columns.on ? SS_DIGITS_CHEB_INV : 0);
    return SS_OK;
}
