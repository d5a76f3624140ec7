// ss_digit_cheb.cu — the Chebyshev column stages of binary64 RLZ grids on the
// tensor cores, by products of digit slices (ss_digit.cu; with at most 48 modes in the
// inverse and 64 levels in the forward direction a digit sum is below 1.31 and 1.75 times 2^24
// for any data, 2^19 rms for random digits).
//
// CA (Γ fold), the CIx recurrence and the DCT-I are linear, so an output column of
// derivative order d is u = M_d b with M_d = IDCT·(D/dscale)^d·Γ composed on the
// host (N × b_kDim).  The column inverse reads the ring stage's quadrant parts as
// they are (64-bit fixed point with one exponent per ring, mode and output),
// forms the four reflected points of each quadrant position by integer
// additions, cuts each column into digits at its own exponent and multiplies by
// the matrix digits, which stay in shared memory.
//
// A fixed-point column is right to 2^-54 of its largest entry, which for ∂z and ∂zz must
// be the largest contribution, not the largest mode: their matrices do not see a column's
// mean (natural ends) and grow with the fourth power of the mode number.  So every column
// k of M_d gives its largest exponent c_k to the data, u = (M_d 2^-c)(2^c b), and f, ∂z
// and ∂zz are cut apart, 7 cuts for the 5 ring outputs.  One cut at f's exponent for all
// three is faster (200 cells, 32 levels, 5 variables, the whole inverse 11.8 against 12.7 ms)
// and loses 2^-55 of the mean, and of the low modes by the fourth power.
//
// Measured on the 200-cell, 32-level, 5-variable FP64 grid: 20.2 ms with FP64 FMAs
// (94% of the FP64 matmul rate), 7.2 ms as digits with loads in line, 4.95 ms with
// the next parts in flight (cp.async), 16 draining warps and the words of a digit
// sum added by wide multiply-adds (shifts and logic run at half rate); 6.0 ms with the
// derivatives cut apart (6.7 before four modes were cut at a time).  Memory
// alone would take 1.4 ms; what is left is the integer work of cutting (five cuts: 8 warps
// without it 3.5 ms) and of rounding 64-bit fixed point to binary64.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "ss_digit.h"
#include "ss_digit_dev.cuh"
#include "ss_grid.h"
#include "ss_internal.h"
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

constexpr int kZ = 32;                      // matrix rows (levels) of one product
constexpr int kZStep = 6 * kZ * 32;         // bytes of a K-step of matrix digits: 6 planes × 32 rows × 16
constexpr int kAStep = 6 * kDigitPlane;     // and of column digits
// Warps: producing, draining (half of them per accumulator), one issuing.  Measured
// on the 200-cell FP64 grid with five cuts: 8 + 16 warps 4.95 ms, 16 + 8 5.34 ms, 8 + 8 5.7 ms;
// with seven, 12 + 16 is 0.1 ms slower than 8 + 16.
constexpr int kProducers = 8, kDrains = 16;
constexpr int kColThreads = (kProducers + kDrains + 1) * 32;
constexpr int kMaxModes = 48;               // three K-steps: what the shared memory holds
constexpr int kMaxZBlocks = 5;              // 160 levels
// Shared memory a CTA may ask for: 227 KB less the static part.  Attribute of both column
// kernels, whatever a grid needs: it is the process's, and grids of other level counts share it.
constexpr size_t kColumnSmem = 232448 - 8192;
// Row-exponent slots: while the producers write those of cut i (at a block's first cut also
// of i + 1 and i + 2), the drain may still read those of cut i − 2 − buffers.
constexpr int kRowExpo = 8;
constexpr int kCuts = kDigitVariants + 2;   // of a block: f for f, ∂z, ∂zz, then ∂λ, ∂λλ, ∂r, ∂rr
constexpr int kUnseen = -(1 << 24);

struct ColumnArgs {
    const void *H;
    double *phys;
    const DigitRing *rings;
    const int *expo;          // [variant][item][ring]
    const uint8_t *M;         // [var][3][zblocks][steps] matrix digits
    const int *mexpo;         // [var][3][32·zblocks]
    const int *weight;        // [var][3][bk] c_k, kUnseen where M_d has no entry for the mode
    const int2 *blocks;       // (ring, first quadrant position) of every 32-position block
    int nblocks;
    int N, bk, nvars, nitems, iDim, steps, zblocks, buffers, raws;
    int64_t jDim, np;
    int *err;
};

__device__ __forceinline__ void producers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kProducers * 32) : "memory"); }
__device__ __forceinline__ void st_global_32B(double *p, const double (&v)[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]) : "memory");
}

// one K-step of a product: D_1..D_6, then D_0, then the rest of digit 0 on the
// first step (as in digit_gemm)
__device__ __forceinline__ void issue_step64(uint32_t tacc, uint32_t sa, uint32_t sb, bool first) {
    const uint64_t bd = operand_desc(sb);
    if (first) {
        mma_f16(tacc + kZ, operand_desc(sa + kDigitPlane), bd, mma_idesc(6 * kZ), 0u);
        mma_f16(tacc, operand_desc(sa), bd, mma_idesc(kZ), 0u);
        mma_f16(tacc + kZ, operand_desc(sa), operand_desc(sb + kZ * 32), mma_idesc(5 * kZ), 1u);
    } else {
        mma_f16(tacc, operand_desc(sa), bd, mma_idesc(6 * kZ), 1u);
        mma_f16(tacc + kZ, operand_desc(sa + kDigitPlane), bd, mma_idesc(6 * kZ), 1u);
    }
#pragma unroll
    for (int i = 2; i < 6; i++)
        mma_f16(tacc + i * kZ, operand_desc(sa + i * kDigitPlane), bd, mma_idesc((7 - i) * kZ), 1u);
}

__device__ __forceinline__ int cut_output(int c) { return c < 3 ? 0 : c - 2; }
__device__ __forceinline__ int cut_matrix(int c) { return c < 3 ? c : 0; }

// grid = (CTAs per variable, variables); a CTA walks (block of 32 quadrant
// positions = 128 columns, cut), cuts fastest
// (kSmall: at most two K-steps)
template <bool kSmall>
__global__ void __launch_bounds__(kColThreads, 1) digit_columns_kernel(ColumnArgs g) {
    extern __shared__ __align__(1024) uint8_t dsm[];
    __shared__ __align__(8) uint64_t afull[2], aempty[2], accf[2], acce[2], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int quit;
    __shared__ volatile int halt[2];  // quit as thread 0 saw it, for all producers
    __shared__ int row_expo[kRowExpo][128];
    __shared__ int mode_expo[2][kMaxModes], weight[3][kMaxModes];
    __shared__ int mode_up[3][kMaxModes];  // mode exponent + c_k + 54 of the cuts of this output
    __shared__ __align__(16) int sE[3 * kZ * kMaxZBlocks];  // row exponents of the matrices, less 53
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int v = blockIdx.y, KS = g.steps, nb = g.buffers;
    const int jobs_bytes = KS * kZStep;
    uint8_t *sM = dsm;                                                   // 3 × zblocks × jobs_bytes
    uint8_t *sA = sM + (size_t)3 * g.zblocks * jobs_bytes;               // nb × KS × 24 KB
    long long *raw = reinterpret_cast<long long *>(sA + (size_t)nb * KS * 6 * kDigitPlane);  // raws × bk × 4 × 32
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) {
            bar_init(&afull[i], kProducers * 32);
            bar_init(&aempty[i], 1);
            bar_init(&accf[i], 1);
            bar_init(&acce[i], kDrains * 16);
        }
        bar_init(&drain, 1);
        quit = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(g.M + (size_t)v * 3 * g.zblocks * jobs_bytes);
        for (int i = threadIdx.x; i < 3 * g.zblocks * jobs_bytes / 16; i += blockDim.x) reinterpret_cast<uint4 *>(sM)[i] = src[i];
    }
    for (int i = threadIdx.x; i < nb * KS * kAStep / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(sA)[i] = make_uint4(0, 0, 0, 0);  // K groups of 8 without modes stay zero
    for (int i = threadIdx.x; i < 3 * g.zblocks * kZ; i += blockDim.x) sE[i] = g.mexpo[(size_t)v * 3 * g.zblocks * kZ + i] - 53;
    for (int i = threadIdx.x; i < 3 * g.bk; i += blockDim.x) weight[i / g.bk][i % g.bk] = g.weight[(size_t)v * 3 * g.bk + i];
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int nitem = blockIdx.x < g.nblocks ? ((g.nblocks - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * kCuts : 0;

    if (warp < kProducers) {
        // ---- producers: parts → points → digits.  The parts of the next output are
        // in flight (cp.async) while this one is cut.
        const long long *H = (const long long *)g.H;
        struct Block {  // this thread's quadrant position: offsets of its four parts from the ring's first row
            int64_t base;
            int o[4], L, ring, flags;  // flags: 1 live, 2 on the axes (Ce, Co at 0 and Ce, So at π/2)
        };
        auto load_block = [&](int item) {
            Block k;
            const int2 blk = g.blocks[blockIdx.x + item * gridDim.x];
            const DigitRing *r = g.rings + blk.x;
            const int n = r->n, m = blk.y + lane;
            const bool edge = r->half == 0 && m == 0;
            k.o[0] = m;
            k.o[1] = r->off[1] + m;
            k.o[2] = edge ? n : r->off[2] + m - r->lo[2];
            k.o[3] = edge ? 4 * n - 1 : r->off[3] + m - r->lo[3];
            k.base = (int64_t)g.bk * r->jofs;
            k.L = r->L;
            k.ring = blk.x;
            k.flags = (m < n ? 1 : 0) | (edge ? 2 : 0);
            return k;
        };
        auto fetch = [&](const Block &k, int var, int slot) {
            const long long *h = H + ((int64_t)var * g.nvars + v) * g.bk * g.jDim + k.base;
            long long *dst = raw + (size_t)slot * g.bk * 128 + lane;
            if (k.flags & 1)
                for (int i = warp; i < g.bk; i += kProducers)
#pragma unroll
                    for (int q = 0; q < 4; q++) cp_async<8>(dst + (i * 4 + q) * 32, h + (int64_t)i * k.L + k.o[q]);
            for (int i = threadIdx.x; i < g.bk; i += kProducers * 32)
                cp_async<4>(&mode_expo[slot][i], g.expo + ((size_t)var * g.nitems + (size_t)v * g.bk + i) * g.iDim + k.ring);
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        Block cur, next;
        if (nitem > 0) {
            next = load_block(0);
            fetch(next, 0, 0);
        }
        const int nr = g.raws;
        int out = 0;  // ring outputs so far
        for (int it = 0; it < nitem; it++) {
            const int cut = it % kCuts, var = cut_output(cut), md = cut_matrix(cut), slot = out % nr;
            const bool last = cut >= 2;  // of this output
            const bool more = it - cut + kCuts < nitem || var + 1 < kDigitVariants;
            long long *pts = raw + (size_t)slot * g.bk * 128;
            if (cut == 0 || cut > 2) {
                if (cut == 0) {
                    cur = next;
                    if (it + kCuts < nitem) next = load_block(it / kCuts + 1);
                }
                const int nd = cut == 0 ? 3 : 1;
                if (threadIdx.x < 128)
                    for (int d = 0; d < nd; d++) row_expo[(it + d) % kRowExpo][threadIdx.x] = 0;
                if (more && nr == 2) {
                    if (var + 1 < kDigitVariants) fetch(cur, var + 1, slot ^ 1);
                    else fetch(next, 0, slot ^ 1);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                producers_sync();
                int mx[3][4] = {};
                for (int i = warp; i < g.bk; i += kProducers) {
                    long long *h = pts + i * 128 + lane;
                    const int e = mode_expo[slot][i];
                    long long p[4] = {0, 0, 0, 0};
                    if (cur.flags & 1) {
                        const long long a = h[0], b = h[32], c = h[64], d = h[96];
                        const long long u = a + b, w = c + d, x = a - b, z = c - d;
                        p[0] = u + w; p[1] = u - w; p[2] = x - z; p[3] = x + z;
                        if (cur.flags & 2) { p[0] = u; p[1] = z; p[2] = x; p[3] = w; }
                    }
                    const bool nan = e == kNanColumn;
                    if (lane < 3) mode_up[lane][i] = nan ? 0 : e + weight[lane][i] + 54;
                    const int w0 = weight[0][i], w1 = weight[1][i], w2 = weight[2][i];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        h[q * 32] = p[q];
                        // |p| ≤ 2^b, |p| 2^(e + c − 1074) ≤ 2^(mx − 1074)
                        const int hi = (int)(p[q] >> 32) ^ (int)(p[q] >> 63);
                        const int eb = (nan ? 0 : e) + (hi ? 64 - __clz(hi) : 32);
                        mx[0][q] = max(mx[0][q], nan ? kNanColumn : eb + w0);
                        if (cut == 0) {
                            mx[1][q] = max(mx[1][q], nan ? kNanColumn : eb + w1);
                            mx[2][q] = max(mx[2][q], nan ? kNanColumn : eb + w2);
                        }
                    }
                }
#pragma unroll
                for (int d = 0; d < 3; d++)
                    if (d < nd) {
#pragma unroll
                        for (int q = 0; q < 4; q++) atomicMax(&row_expo[(it + d) % kRowExpo][q * 32 + lane], mx[d][q]);
                    }
                // the producers leave together, on one thread's word: one that gave up waiting alone would
                // be missed at the barrier for good
                if (threadIdx.x == 0) halt[out & 1] = quit;
                producers_sync();
                if (halt[out & 1]) break;
            }
            const int buf = it % nb;
            const bool ok = bar_wait(&aempty[buf], ((it / nb) & 1) ^ 1, &quit);  // if not: quit is set
            uint8_t *A = sA + (size_t)buf * KS * 6 * kDigitPlane;
            const int row = threadIdx.x & 127;
            const int er = min(row_expo[it % kRowExpo][row], 1 << 28);
            // four modes at a time: 22 modes are three such cuts of every thread
            for (int kq = threadIdx.x >> 7; ok && kq < (g.bk + 3) / 4; kq += kProducers / 4) {
                unsigned long long U[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int mode = kq * 4 + i;
                    long long X = 0;
                    if (mode < g.bk) {
                        X = pts[mode * 128 + row];
                        const int s = mode_up[md][mode] - er;  // |V 2^s| ≤ 2^54
                        if (s > 0) X <<= min(s, 63);
                        else if (s < 0) X = s > -63 ? ((X >> (-s - 1)) + 1) >> 1 : 0;
                    }
                    U[i] = kDigitBias + (unsigned long long)X;
                }
                uint2 w[6];
                planes4(U, w);
                uint8_t *dst = A + (kq >> 2) * 6 * kDigitPlane + (row >> 3) * 256 + ((kq >> 1) & 1) * 128 + (row & 7) * 16 + (kq & 1) * 8;
#pragma unroll
                for (int i = 0; i < 6; i++) *reinterpret_cast<uint2 *>(dst + i * kDigitPlane) = w[i];
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (ok) bar_arrive(&afull[buf]);
            if (!last) continue;
            producers_sync();  // these points may be overwritten
            if (more && nr == 1) {
                if (var + 1 < kDigitVariants) fetch(cur, var + 1, 0);
                else fetch(next, 0, 0);
            }
            out++;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else if (warp == kProducers + kDrains) {
        // ---- issuer
        if (lane == 0) {
            bool ok = true;
            uint32_t job = 0;
            for (int it = 0; ok && it < nitem; it++) {
                const int buf = it % nb;
                if (!(ok = bar_wait(&afull[buf], (it / nb) & 1, &quit))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t sa0 = smem_addr(sA) + buf * KS * 6 * kDigitPlane;
                const int q0 = cut_matrix(it % kCuts) * g.zblocks;
                for (int q = q0; ok && q < q0 + g.zblocks; q++, job++) {
                    const int t = job & 1;
                    if (!(ok = bar_wait(&acce[t], ((job >> 1) & 1) ^ 1, &quit))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t tacc = tmem + t * 256;
                    for (int k = 0; k < KS; k++) {
                        const uint32_t sa = sa0 + k * 6 * kDigitPlane, sb = smem_addr(sM) + (q * KS + k) * kZStep;
                        issue_step64(tacc, sa, sb, k == 0);
                    }
                    mma_commit(&accf[t]);
                }
                if (ok) mma_commit(&aempty[buf]);
            }
            if (!ok) {
                int never = 0;
                mma_commit(&drain);
                bar_wait(&drain, 0, &never);
            }
        }
    } else {
        // ---- drain: eight warps per accumulator; thread = (column, 16 levels)
        const int mine = (warp - kProducers) >> 3;  // the accumulator, i.e. the parity of the jobs
        const int zh = ((warp >> 2) & 1) * 16;
        const int quad = warp & 3, row = quad * 32 + lane;
        const uint32_t tacc = tmem + ((uint32_t)(quad * 32) << 16) + mine * 256 + zh;
        const bool vec = g.N % 4 == 0;
        uint32_t job = 0;
        bool ok = true;
        for (int it = 0; ok && it < nitem; it++) {
            const int cut = it % kCuts, var = cut_output(cut), d = cut_matrix(cut);
            const int2 blk = g.blocks[blockIdx.x + it / kCuts * gridDim.x];
            const DigitRing *r = g.rings + blk.x;
            const int n = r->n, L = r->L, hf = r->half, m = blk.y + lane;
            const bool edge = hf == 0 && m == 0, live = m < n;
            int p = quad == 0 ? m : (quad == 1 ? 4 * n - hf - m : (quad == 2 ? 2 * n - hf - m : 2 * n + m));
            if (edge) p = quad == 0 ? 0 : (quad == 1 ? 3 * n : (quad == 2 ? 2 * n : n));
            int l = p - r->shift;
            if (l < 0) l += L;
            if (l >= L) l -= L;
            double *const col = g.phys + (size_t)v * g.np + (r->jofs + l) * g.N;
            for (int zb = 0; ok && zb < g.zblocks; zb++, job++) {
                if ((int)(job & 1) != mine) continue;
                const int z0 = zb * kZ + zh;
                const int slot = var == 0 ? (d == 0 ? 0 : 4 + d) : (var == 1 ? 3 : (var == 2 ? 4 : var - 2));
                double *dst = col + (size_t)slot * g.nvars * g.np + z0;
                if (!(ok = __all_sync(0xffffffffu, bar_wait(&accf[mine], (job >> 1) & 1, &quit)))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int er = row_expo[it % kRowExpo][row];
                const int *me = sE + (d * g.zblocks + zb) * kZ + zh;
                // rolled: the instruction cache serves all three roles
#pragma unroll 1
                for (int c0 = 0; c0 < 16; c0 += 4) {
                    float D[7][4];
#pragma unroll
                    for (int s = 0; s < 7; s++) tmem_ld4(tacc + s * kZ + c0, D[s]);
                    const int4 e4 = *reinterpret_cast<const int4 *>(me + c0);
                    tmem_wait_ld();
                    if (c0 == 12) {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        bar_arrive(&acce[mine]);
                    }
                    const int ze[4] = {e4.x, e4.y, e4.z, e4.w};
                    double o[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        unsigned long long V = 0ull - Combine<kSmall>::kOffset;
                        Combine<kSmall>::add(V, D[0][c], D[1][c], D[2][c], D[3][c], D[4][c], D[5][c], D[6][c]);
                        o[c] = fixed_to_double((long long)V, er + ze[c]);  // V 2^(er − 1074 + mexpo − 53)
                        if (er == kNanColumn) o[c] = __longlong_as_double(0x7ff8000000000000ll);
                    }
                    if (live) {
                        if (vec) {
                            if (z0 + c0 < g.N) st_global_32B(dst + c0, o);
                        } else {
#pragma unroll
                            for (int c = 0; c < 4; c++)
                                if (z0 + c0 + c < g.N) dst[c0 + c] = o[c];
                        }
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && quit) *g.err = 1;
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ------------------------------------------------------------ forward columns
// CBtransform! of binary64 grids: the first b_kDim modes of 128 consecutive columns
// per tile.  A column's levels are contiguous, so 4 or 8 neighbouring lanes hold
// 8 levels each, find the column's exponent by shuffles and cut in registers.
// Two operand buffers of 24 KB a K-step and the matrix leave room for grids of up to 48
// levels, and of up to 64 with at most 32 modes; longer columns keep the FMA kernel.
// Measured: 200 cells, 32 levels, 5 variables 2.60 ms with FP64 FMAs → 0.81 ms (the bytes
// alone take 0.23 ms), 37 cells, 20 levels, 3 variables 37 → 25 µs; bound by cutting and
// combining.  The error against 64-bit sums is no larger than the FMA kernel's.
struct ForwardColumnArgs {
    const double *phys;       // slot 1
    double *C;                // [variable][ring][mode][ring point]
    const RingDesc *rings;
    const int *col_ring;
    const uint8_t *M;         // [var][mode blocks][steps] matrix digits
    const int *mexpo;         // [var][32·mode blocks]
    int64_t col0, col1, np, jDim;
    int N, bk, steps, blocks, group;
    int *err;
};

__global__ void __launch_bounds__(kColThreads, 1) digit_columns_forward_kernel(ForwardColumnArgs g) {
    extern __shared__ __align__(1024) uint8_t dsm[];
    __shared__ __align__(8) uint64_t afull[2], aempty[2], accf[2], acce[2], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int quit;
    __shared__ int row_expo[kRowExpo][128];
    __shared__ __align__(16) int sE[kZ * kMaxZBlocks];  // row exponents of the matrix, less 1
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int v = blockIdx.y, KS = g.steps;
    uint8_t *sM = dsm, *sA = sM + (size_t)g.blocks * KS * kZStep;  // matrix, then 2 operand buffers
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) {
            bar_init(&afull[i], kProducers * 32);
            bar_init(&aempty[i], 1);
            bar_init(&accf[i], 1);
            bar_init(&acce[i], kDrains * 16);
        }
        bar_init(&drain, 1);
        quit = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(g.M + (size_t)v * g.blocks * KS * kZStep);
        for (int i = threadIdx.x; i < g.blocks * KS * kZStep / 16; i += blockDim.x) reinterpret_cast<uint4 *>(sM)[i] = src[i];
    }
    for (int i = threadIdx.x; i < 2 * KS * kAStep / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(sA)[i] = make_uint4(0, 0, 0, 0);  // levels beyond N stay zero
    for (int i = threadIdx.x; i < g.blocks * kZ; i += blockDim.x) sE[i] = g.mexpo[(size_t)v * g.blocks * kZ + i] - 1;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int64_t ntile = (g.col1 - g.col0 + 127) / 128;
    const int nitem = (int)((ntile - blockIdx.x + gridDim.x - 1) / gridDim.x);

    if (warp < kProducers) {
        const int G = g.group, per = 256 / G;  // lanes of a column, columns of a sweep
        const int kg = threadIdx.x % G, z0 = kg * 8;
        const bool pairs = g.N % 2 == 0;
        auto load = [&](int64_t c, double (&x)[8]) {
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = 0.0;
            if (c >= g.col1) return;
            const double *src = g.phys + (size_t)v * g.np + c * g.N + z0;
            if (pairs) {
#pragma unroll
                for (int i = 0; i < 8; i += 2)
                    if (z0 + i < g.N) {
                        const double2 t = *reinterpret_cast<const double2 *>(src + i);
                        x[i] = t.x; x[i + 1] = t.y;
                    }
            } else {
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (z0 + i < g.N) x[i] = src[i];
            }
        };
        bool ok = true;
        double x[8], next[8];
        load(g.col0 + blockIdx.x * 128ll + threadIdx.x / G, next);
        for (int it = 0; ok && it < nitem; it++) {
            const int64_t c0 = g.col0 + (blockIdx.x + (int64_t)it * gridDim.x) * 128;
            const int buf = it & 1;
            uint8_t *A = sA + (size_t)buf * KS * kAStep;
            for (int r0 = 0; r0 < 128; r0 += per) {
                const int row = r0 + threadIdx.x / G;
#pragma unroll
                for (int i = 0; i < 8; i++) x[i] = next[i];
                // the next sweep's levels (of this tile or the first of the next) arrive while these are cut
                const bool last = r0 + per >= 128;
                const int64_t ahead = last ? (it + 1 < nitem ? c0 + 128ll * gridDim.x + threadIdx.x / G : g.col1) : c0 + row + per;
                load(ahead, next);
                uint32_t mx = 0;
#pragma unroll
                for (int i = 0; i < 8; i++) mx = max(mx, (uint32_t)__double2hiint(x[i]) & 0x7fffffffu);
                for (int o = 1; o < G; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const int eb = (int)(mx >> 20), e = eb == 0x7ff ? kNanColumn : max(eb, 1);
                unsigned long long U[8];
#pragma unroll
                for (int i = 0; i < 8; i++) U[i] = kDigitBias + (unsigned long long)(e == kNanColumn ? 0ll : fixed_point<54>(x[i], e));
                uint4 w[6];
                planes8(U, w);
                // a warp decides as one: its lanes exchange values in the next sweep
                if (r0 == 0 && !(ok = __all_sync(0xffffffffu, bar_wait(&aempty[buf], ((it >> 1) & 1) ^ 1, &quit)))) break;
                if (kg == 0) row_expo[it % kRowExpo][row] = e;
                if (kg < 2 * KS) {
                    uint8_t *dst = A + (kg >> 1) * kAStep + (row >> 3) * 256 + (kg & 1) * 128 + (row & 7) * 16;
#pragma unroll
                    for (int i = 0; i < 6; i++) *reinterpret_cast<uint4 *>(dst + i * kDigitPlane) = w[i];
                }
            }
            if (!ok) break;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            bar_arrive(&afull[buf]);
        }
    } else if (warp == kProducers + kDrains) {
        if (lane == 0) {
            bool ok = true;
            uint32_t job = 0;
            for (int it = 0; ok && it < nitem; it++) {
                const int buf = it & 1;
                if (!(ok = bar_wait(&afull[buf], (it >> 1) & 1, &quit))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int q = 0; ok && q < g.blocks; q++, job++) {
                    const int t = job & 1;
                    if (!(ok = bar_wait(&acce[t], ((job >> 1) & 1) ^ 1, &quit))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int k = 0; k < KS; k++)
                        issue_step64(tmem + t * 256, smem_addr(sA) + (buf * KS + k) * kAStep, smem_addr(sM) + (q * KS + k) * kZStep, k == 0);
                    mma_commit(&accf[t]);
                }
                if (ok) mma_commit(&aempty[buf]);
            }
            if (!ok) {
                int never = 0;
                mma_commit(&drain);
                bar_wait(&drain, 0, &never);
            }
        }
    } else {
        const int mine = (warp - kProducers) >> 3;
        const int zh = ((warp >> 2) & 1) * 16;
        const int quad = warp & 3, row = quad * 32 + lane;
        const uint32_t tacc = tmem + ((uint32_t)(quad * 32) << 16) + mine * 256 + zh;
        uint32_t job = 0;
        bool ok = true;
        for (int it = 0; ok && it < nitem; it++) {
            const int64_t c = g.col0 + (blockIdx.x + (int64_t)it * gridDim.x) * 128 + row;
            const bool live = c < g.col1;
            const RingDesc *r = g.rings + (live ? g.col_ring[c] : 0);
            const int64_t L = r->L;
            double *const out = g.C + (size_t)v * g.bk * g.jDim + (int64_t)g.bk * r->jofs + (c - r->jofs);
            for (int q = 0; ok && q < g.blocks; q++, job++) {
                if ((int)(job & 1) != mine) continue;
                if (!(ok = __all_sync(0xffffffffu, bar_wait(&accf[mine], (job >> 1) & 1, &quit)))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int er = row_expo[it % kRowExpo][row];
                const int m0 = q * kZ + zh;
#pragma unroll 1
                for (int k0 = 0; k0 < 16 && m0 + k0 < g.bk; k0 += 4) {
                    float D[7][4];
#pragma unroll
                    for (int s = 0; s < 7; s++) tmem_ld4(tacc + s * kZ + k0, D[s]);
                    tmem_wait_ld();
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        unsigned long long V = 0ull - Combine<false>::kOffset;
                        Combine<false>::add(V, D[0][k], D[1][k], D[2][k], D[3][k], D[4][k], D[5][k], D[6][k]);
                        double o = fixed_to_double((long long)V, er + sE[m0 + k0 + k]);  // V 2^(er − 1022 + mexpo − 53)
                        if (er == kNanColumn) o = __longlong_as_double(0x7ff8000000000000ll);
                        if (live && m0 + k0 + k < g.bk) out[(int64_t)(m0 + k0 + k) * L] = o;
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                bar_arrive(&acce[mine]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && quit) *g.err = 1;
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ------------------------------------------------------------ host
// balanced digits of x·2^(53 − e), |x| < 2^e (53-bit fixed point), most significant first
static void host_digits(double x, int e, int (&d)[6]) {
    long long X = std::llrint(std::ldexp(x, 53 - e));
    for (int i = 5; i > 0; i--) {
        long long q = ((X + 256) & 511) - 256;
        d[i] = (int)q;
        X = (X - q) / 512;
    }
    d[0] = (int)X;
}

static size_t column_smem(int steps, int zblocks, int bk, int buffers, int raws) {
    return (size_t)3 * zblocks * steps * kZStep + (size_t)buffers * steps * 6 * kDigitPlane + (size_t)raws * bk * 128 * 8;
}

static size_t forward_smem(int steps, int blocks) {
    return (size_t)blocks * steps * kZStep + (size_t)2 * steps * kAStep;
}

static int32_t build_forward(ss_grid *g, const std::vector<ChebHost> &cheb) {
    DigitColumns &Q = g->digit.columns;
    const int N = (int)g->d.kDim, bk = (int)g->d.b_kDim, nv = (int)g->d.nvars;
    Q.fsteps = (N + 15) / 16;
    Q.fblocks = (bk + kZ - 1) / kZ;
    Q.fgroup = N <= 32 ? 4 : 8;
    if (Q.fsteps > 4 || Q.fblocks > kMaxZBlocks || forward_smem(Q.fsteps, Q.fblocks) > kColumnSmem) return SS_OK;
    const int job = Q.fsteps * kZStep;
    std::vector<uint8_t> M((size_t)nv * Q.fblocks * job, 0);
    std::vector<int> E((size_t)nv * Q.fblocks * kZ, 0);
    for (int v = 0; v < nv; v++) {
        const ChebHost &c = cheb[v];
        if (v > 0) {  // the forward matrix knows no ends: one for all variables
            std::copy_n(M.begin(), (size_t)Q.fblocks * job, M.begin() + (size_t)v * Q.fblocks * job);
            std::copy_n(E.begin(), (size_t)Q.fblocks * kZ, E.begin() + (size_t)v * Q.fblocks * kZ);
            continue;
        }
        for (int k = 0; k < bk; k++) {
            std::vector<double> row(N, 0.0);
            double top = 0.0;
            for (int j = 0; j < c.half; j++) {  // folded over j ↔ N − 1 − j: even k +, odd k −
                const double w = c.fwd[(size_t)k * c.half + j];
                row[j] = w;
                if (N - 1 - j != j) row[N - 1 - j] = k % 2 ? -w : w;
                top = std::max(top, std::fabs(w));
            }
            int e = 0;
            if (top > 0.0) std::frexp(top, &e);
            const int kb = k / kZ, kr = k % kZ;
            E[((size_t)v * Q.fblocks + kb) * kZ + kr] = e;
            uint8_t *dst = M.data() + ((size_t)v * Q.fblocks + kb) * job;
            for (int j = 0; j < N; j++) {
                int dg[6];
                host_digits(row[j], e, dg);
                for (int q = 0; q < 6; q++) {
                    const __half h = __float2half_rn((float)dg[q]);
                    const int rr = q * kZ + kr, kk = j % 16;
                    std::memcpy(dst + (j / 16) * kZStep + (rr >> 3) * 256 + (kk >> 3) * 128 + (rr & 7) * 16 + (kk & 7) * 2, &h, 2);
                }
            }
        }
    }
    DigitBlock blk;
    blk.put(&Q.fM, M);
    blk.put(&Q.fexpo, E);
    if (!blk.build(g->allocs)) return SS_OK;
    CUDA_TRY(cudaFuncSetAttribute(digit_columns_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kColumnSmem));
    Q.fon = true;
    return SS_OK;
}

static int32_t build_inverse(ss_grid *g, const std::vector<ChebHost> &cheb) {
    DigitPlan &P = g->digit;
    const int N = (int)g->d.kDim, bk = (int)g->d.b_kDim, nv = (int)g->d.nvars;
    DigitColumns &Q = P.columns;
    Q.steps = (bk + 15) / 16;
    Q.zblocks = (N + kZ - 1) / kZ;
    if (bk > kMaxModes || Q.zblocks > kMaxZBlocks) return SS_OK;
    // two operand buffers and two input buffers where they fit, then fewer
    const int shapes[4][2] = {{2, 2}, {1, 2}, {2, 1}, {1, 1}};
    Q.buffers = 0;
    for (const auto &s : shapes)
        if (!Q.buffers && column_smem(Q.steps, Q.zblocks, bk, s[0], s[1]) <= kColumnSmem) { Q.buffers = s[0]; Q.raws = s[1]; }
    if (!Q.buffers) return SS_OK;
    const int job = Q.steps * kZStep;
    std::vector<uint8_t> M((size_t)nv * 3 * Q.zblocks * job, 0);
    std::vector<int> E((size_t)nv * 3 * Q.zblocks * kZ, 0), W((size_t)nv * 3 * bk, kUnseen);
    for (int v = 0; v < nv; v++) {
        const ChebHost &c = cheb[v];
        int like = 0;  // the first variable with the same ends
        while (g->bcb[like] != g->bcb[v] || g->bct[like] != g->bct[v]) like++;
        if (like < v) {
            const size_t m = (size_t)3 * Q.zblocks * job, e = (size_t)3 * Q.zblocks * kZ, w = (size_t)3 * bk;
            std::copy_n(M.begin() + like * m, m, M.begin() + v * m);
            std::copy_n(E.begin() + like * e, e, E.begin() + v * e);
            std::copy_n(W.begin() + like * w, w, W.begin() + v * w);
            continue;
        }
        const int ne = (N + 1) / 2, no = std::max(N / 2, 1);
        std::vector<double> X((size_t)N * bk, 0.0), Y((size_t)N * bk);
        for (int k = 0; k < N; k++)
            for (int i = 0; i < bk; i++) {
                double s = k == i ? 1.0 : 0.0;
                for (int p = 0; p < c.nrank; p++) s += c.gv[(size_t)p * N + k] * c.gu[(size_t)p * bk + i];
                X[(size_t)k * bk + i] = s;
            }
        for (int d = 0; d < 3; d++) {
            if (d > 0) {
                for (int k = 0; k < N; k++)
                    for (int i = 0; i < bk; i++) {
                        double s = 0.0;
                        for (int m = k + 1; m < N; m += 2) s += 2.0 * m * X[(size_t)m * bk + i];
                        Y[(size_t)k * bk + i] = s / c.dscale;
                    }
                X.swap(Y);
            }
            std::vector<double> M_d((size_t)N * bk);
            for (int z = 0; z < N; z++) {
                const int j = std::min(z, N - 1 - z);  // inv_e, inv_o hold the first half of the levels
                const double so = z == j ? 1.0 : -1.0;
                for (int i = 0; i < bk; i++) {
                    double a = 0.0, b = 0.0;
                    for (int k = 0; k < N; k += 2) a += c.inv_e[(size_t)j * ne + k / 2] * X[(size_t)k * bk + i];
                    for (int k = 1; k < N; k += 2) b += c.inv_o[(size_t)j * no + k / 2] * X[(size_t)k * bk + i];
                    M_d[(size_t)z * bk + i] = a + so * b;
                }
            }
            int *w = W.data() + ((size_t)v * 3 + d) * bk;
            for (int i = 0; i < bk; i++) {
                double top = 0.0;
                for (int z = 0; z < N; z++) top = std::max(top, std::fabs(M_d[(size_t)z * bk + i]));
                if (top > 0.0) std::frexp(top, &w[i]);
            }
            for (int z = 0; z < N; z++) {
                double top = 0.0;
                std::vector<double> row(bk, 0.0);
                for (int i = 0; i < bk; i++) {
                    if (w[i] != kUnseen) row[i] = std::ldexp(M_d[(size_t)z * bk + i], -w[i]);
                    top = std::max(top, std::fabs(row[i]));
                }
                int e = 0;
                if (top > 0.0) std::frexp(top, &e);
                const int zb = z / kZ, zr = z % kZ;
                E[(((size_t)v * 3 + d) * Q.zblocks + zb) * kZ + zr] = e;
                uint8_t *dst = M.data() + (((size_t)v * 3 + d) * Q.zblocks + zb) * job;
                for (int i = 0; i < bk; i++) {
                    int dg[6];
                    host_digits(row[i], e, dg);
                    for (int q = 0; q < 6; q++) {
                        const __half h = __float2half_rn((float)dg[q]);
                        const int rr = q * kZ + zr, kk = i % 16;
                        std::memcpy(dst + (i / 16) * kZStep + (rr >> 3) * 256 + (kk >> 3) * 128 + (rr & 7) * 16 + (kk & 7) * 2, &h, 2);
                    }
                }
            }
        }
    }
    // blocks of 32 quadrant positions, rings ascending (a radial chunk is a contiguous run)
    std::vector<int2> blocks;
    Q.first.assign(1, 0);
    for (int r = 0; r < g->d.iDim; r++) {
        const int n = r + 1 + g->pOL + 1;
        for (int m = 0; m < n; m += 32) blocks.push_back(make_int2(r, m));
        Q.first.push_back((int)blocks.size());
    }
    DigitBlock blk;
    blk.put(&Q.M, M);
    blk.put(&Q.mexpo, E);
    blk.put(&Q.weight, W);
    blk.put(&Q.blocks, blocks);
    if (!blk.build(g->allocs)) return SS_OK;
    CUDA_TRY(cudaFuncSetAttribute(Q.steps <= 2 ? digit_columns_kernel<true> : digit_columns_kernel<false>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kColumnSmem));
    Q.on = true;
    return SS_OK;
}

int32_t digit_columns_build(ss_grid *g, const std::vector<ChebHost> &cheb) {
    if (!g->digit.on || !g->rlz || g->tl != TL_F64) return SS_OK;
    const int32_t rc = build_forward(g, cheb);
    return rc ? rc : build_inverse(g, cheb);
}

int32_t digit_columns_forward(ss_grid *g, cudaStream_t st, int64_t col0, int64_t col1) {
    if (col1 <= col0) return SS_OK;
    const DigitColumns &Q = g->digit.columns;
    const ss_dims &d = g->d;
    ForwardColumnArgs A{};
    A.phys = (const double *)g->phys; A.C = (double *)g->C; A.rings = g->d_rings; A.col_ring = g->d_col_ring;
    A.M = Q.fM; A.mexpo = Q.fexpo; A.col0 = col0; A.col1 = col1; A.np = d.n_physical; A.jDim = d.jDim;
    A.N = (int)d.kDim; A.bk = (int)d.b_kDim; A.steps = Q.fsteps; A.blocks = Q.fblocks; A.group = Q.fgroup; A.err = g->digit.err;
    const int64_t tiles = (col1 - col0 + 127) / 128;
    const int per = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, g->sms / (int)d.nvars));
    digit_columns_forward_kernel<<<dim3(per, (unsigned)d.nvars), kColThreads, forward_smem(Q.fsteps, Q.fblocks), st>>>(A);
    CUDA_TRY(cudaGetLastError());
    return SS_OK;
}

int32_t digit_columns_inverse(ss_grid *g, cudaStream_t st, int chunk) {
    const DigitPlan &P = g->digit;
    const DigitColumns &Q = P.columns;
    const ss_dims &d = g->d;
    const int r0 = chunk < 0 ? 0 : g->chunk_r0[chunk], r1 = chunk < 0 ? (int)d.iDim : g->chunk_r0[chunk + 1];
    ColumnArgs A{};
    A.H = g->H; A.phys = (double *)g->phys; A.rings = P.rings; A.expo = P.expo;
    A.M = Q.M; A.mexpo = Q.mexpo; A.weight = Q.weight; A.blocks = Q.blocks + Q.first[r0]; A.nblocks = Q.first[r1] - Q.first[r0];
    A.N = (int)d.kDim; A.bk = (int)d.b_kDim; A.nvars = (int)d.nvars; A.nitems = g->nitems; A.iDim = (int)d.iDim;
    A.steps = Q.steps; A.zblocks = Q.zblocks; A.buffers = Q.buffers; A.raws = Q.raws; A.jDim = d.jDim; A.np = d.n_physical; A.err = P.err;
    const int per = std::max(1, std::min(A.nblocks, g->sms / (int)d.nvars));
    const size_t smem = column_smem(Q.steps, Q.zblocks, A.bk, Q.buffers, Q.raws);
    const dim3 grid(per, (unsigned)d.nvars);
    if (Q.steps <= 2) digit_columns_kernel<true><<<grid, kColThreads, smem, st>>>(A);
    else digit_columns_kernel<false><<<grid, kColThreads, smem, st>>>(A);
    CUDA_TRY(cudaGetLastError());
    return SS_OK;
}

}  // namespace ss
