// ss_digit_dev.cuh — device pieces shared by the digit-slice kernels: cutting
// values into digits, the bounded barriers, the tensor-core instructions and the
// recombination of the digit sums.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "ss_digit.h"

namespace ss {

// ------------------------------------------------------------ digits
// two unsigned fields of at most 1024 minus `bias`, exactly, as a half2
__device__ __forceinline__ uint32_t half_pair(uint32_t a, uint32_t b, uint32_t bias) {
    const uint32_t v = 0x64006400u + a + (b << 16);  // 1024 + field in each half
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&v), *reinterpret_cast<const __half2 *>(&bias));
    return *reinterpret_cast<const uint32_t *>(&h);
}
// X + bias, |X| ≤ 2^54: five low fields of 9 bits are the balanced digits + 256,
// the rest is the leading digit + 512
constexpr unsigned long long kDigitBias =
    256ull * ((1ull << 0) + (1ull << 9) + (1ull << 18) + (1ull << 27) + (1ull << 36)) + (512ull << 45);

// |x| < 2^(emax − 1022) as `bits`-bit fixed point (bits ≤ 61), rounded
template <int kBits>
__device__ __forceinline__ long long fixed_point(double x, int emax) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int e = (int)((u >> 52) & 0x7ff);
    unsigned long long m = u & 0xfffffffffffffull;
    if (e > 0) m |= 0x10000000000000ull;
    const int r = min(emax - max(e, 1), 63);
    m = (((m << (kBits - 52)) >> r) + 1) >> 1;
    return (long long)u < 0 ? -(long long)m : (long long)m;
}
// digit planes of 8 consecutive K entries: out[i] = 16 bytes of plane i, most significant first
__device__ __forceinline__ void planes8(const unsigned long long (&U)[8], uint4 (&out)[6]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const int sh = 45 - 9 * i;
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint32_t a = (uint32_t)(U[2 * q] >> sh), b = (uint32_t)(U[2 * q + 1] >> sh);
            if (i > 0) { a &= 511u; b &= 511u; }
            w[q] = half_pair(a, b, i > 0 ? 0x65006500u : 0x66006600u);  // 1024 + 256 or 512
        }
        out[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
// binary32: x·2^-E = (d0 + d1/1024 + d2/1024²)/256
__device__ __forceinline__ void planes8(const float (&x)[8], uint4 (&out)[3]) {
    constexpr float M = 12582912.f;  // 1.5·2^23: adding it rounds to the nearest integer
    uint32_t w[3][4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        float d[3][2];
#pragma unroll
        for (int p = 0; p < 2; p++) {
            float v = x[2 * q + p];
            d[0][p] = (v + M) - M;
            v = (v - d[0][p]) * 1024.f;
            d[1][p] = (v + M) - M;
            v = (v - d[1][p]) * 1024.f;
            d[2][p] = (v + M) - M;
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const __half2 h = __floats2half2_rn(d[i][0], d[i][1]);
            w[i][q] = *reinterpret_cast<const uint32_t *>(&h);
        }
    }
#pragma unroll
    for (int i = 0; i < 3; i++) out[i] = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

// x scaled by 2^s, |s| ≤ 300 (two exact factors: 2^s itself may leave the type's range)
__device__ __forceinline__ float pow2f(int s) { return __int_as_float((s + 127) << 23); }
__device__ __forceinline__ float scale2(float x, int s) {
    const int a = s / 2;
    return (x * pow2f(a)) * pow2f(s - a);
}

// ------------------------------------------------------------ tensor cores
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// K-major no-swizzle operand: core matrices 128 B apart along K, 8-row groups 256 B apart
__device__ __forceinline__ uint64_t operand_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46);
}
// kind::f16, binary16 operands, binary32 accumulators, M = 128
__host__ __device__ constexpr uint32_t mma_idesc(int N) { return (1u << 4) | ((uint32_t)(N >> 3) << 17) | (8u << 24); }
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void bar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ long long now_ns() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
constexpr long long kDigitWaitNs = 2000000000LL;
// bounded wait; false once it has lasted two seconds or another role has given up
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity, volatile int *quit) {
    if (bar_try(bar, parity)) return true;
    const long long t0 = now_ns();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (bar_try(bar, parity)) return true;
        if (*quit) return false;
        if (now_ns() - t0 > kDigitWaitNs) {
            *quit = 1;
            return false;
        }
    }
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Σ_s D_s 2^(36−9s) (D_5, D_6 rounded): the D_s are integers of up to 2^26; each is
// cut at 2^9 by a fused multiply-add with 1.5·2^23 (which leaves an integer in the
// low mantissa bits), the high part joining the next sum, so that every word is
// far inside the 23-bit range
__device__ __forceinline__ long long combine(const float D0, const float D1, const float D2, const float D3,
                                             const float D4, const float D5, const float D6) {
    constexpr float M = 12582912.f;
    constexpr int C = 0x4B400000;
    const float b5 = fmaf(fmaf(D6, 0x1p-9f, D5), 0x1p-9f, M);
    const float m4 = fmaf(D4, 0x1p-9f, M), b4 = fmaf(m4 - M, -512.f, D4) + b5;
    const float m3 = fmaf(D3, 0x1p-9f, M), b3 = fmaf(m3 - M, -512.f, D3) + m4;
    const float m2 = fmaf(D2, 0x1p-9f, M), b2 = fmaf(m2 - M, -512.f, D2) + m3;
    const float m1 = fmaf(D1, 0x1p-9f, M), b1 = fmaf(m1 - M, -512.f, D1) + m2;
    const float m0 = fmaf(D0, 0x1p-9f, M), b0 = fmaf(m0 - M, -512.f, D0) + m1;
    const int u0 = (__float_as_int(b0) - C) * 512 + (__float_as_int(b1) - C);
    const int u1 = (__float_as_int(b2) - C) * 512 + (__float_as_int(b3) - C);
    return ((long long)(__float_as_int(m0) - C) << 45) + ((long long)u0 << 27) + ((long long)u1 << 9) +
           (long long)(__float_as_int(b4) - C);
}

// binary64 V·2^(expo − 1074), rounded to nearest even; V = 0 gives 0
__device__ __forceinline__ double fixed_to_double(long long V, int expo) {
    if (V == 0) return 0.0;
    const unsigned long long a = V < 0 ? 0ull - (unsigned long long)V : (unsigned long long)V;
    const int lz = __clzll((long long)a);
    const int ef = expo + 12 - lz;
    if (ef < 1 || ef > 2045) {  // leaves the normal range: two exact factors
        const int s = expo - 1074, h = s / 2;
        return scalbn(scalbn((double)V, h), s - h);
    }
    const unsigned long long n = a << lz;
    const unsigned long long mant = (n >> 11) + (((n & 0x7ffull) + ((n >> 11) & 1ull)) > 0x400ull ? 1ull : 0ull);
    const unsigned long long bits = ((unsigned long long)(ef - 1) << 52) + mant;
    return __longlong_as_double((long long)(V < 0 ? bits | 0x8000000000000000ull : bits));
}

}  // namespace ss
