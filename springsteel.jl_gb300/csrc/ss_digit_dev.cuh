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
// Two unsigned fields of at most 1024 minus `bias` as a half2, exactly.  A matrix
// digit is the integer itself (1024 + field, less 1024 + bias); a data digit is
// its 2^-24 multiple: the field read as a binary16 subnormal, which needs no
// exponent bits set.
// `mask`: the fields' bits in a and b, cut from both halves at once.
template <bool kMatrix>
__device__ __forceinline__ uint32_t half_pair(uint32_t a, uint32_t b, uint32_t mask, uint32_t bias) {
    const uint32_t off = kMatrix ? 0x64006400u : 0u;
    const uint32_t v = off + (__byte_perm(a, b, 0x5410) & mask), w = off + bias;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&v), *reinterpret_cast<const __half2 *>(&w));
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
template <bool kMatrix = false>
__device__ __forceinline__ void planes8(const unsigned long long (&U)[8], uint4 (&out)[6]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const int sh = 45 - 9 * i;
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            w[q] = half_pair<kMatrix>((uint32_t)(U[2 * q] >> sh), (uint32_t)(U[2 * q + 1] >> sh), i > 0 ? 0x01ff01ffu : 0xffffffffu,
                                      i > 0 ? 0x01000100u : 0x02000200u);
        }
        out[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
// and of 4
__device__ __forceinline__ void planes4(const unsigned long long (&U)[4], uint2 (&out)[6]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const int sh = 45 - 9 * i;
        uint32_t w[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            w[q] = half_pair<false>((uint32_t)(U[2 * q] >> sh), (uint32_t)(U[2 * q + 1] >> sh), i > 0 ? 0x01ff01ffu : 0xffffffffu,
                                    i > 0 ? 0x01000100u : 0x02000200u);
        }
        out[i] = make_uint2(w[0], w[1]);
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
__device__ __forceinline__ void tmem_ld4(uint32_t addr, float (&v)[4]) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// acc += Σ_s D_s 2^(36−9s) + kOffset (D_5, D_6 rounded).  The D_s arrive as 2^-24
// multiples (data digits) of integers of up to 2^26; each is cut at 2^9 by a fused
// multiply-add with 1.5·2^23, which leaves an integer in the low mantissa bits,
// the high part joining the next sum, so that every word is far inside the 23-bit
// range.  The words are added as raw bits (32-bit wide multiply-adds run at full
// rate here, shifts and logic at half): the constant they carry is kOffset, taken
// off once per result.  kSmall: |D_0| ≤ 2^22 (at most 32 products) needs no cut.
template <bool kSmall>
struct Combine {
    static constexpr unsigned long long kMagic = 0x4B400000ull;  // bits of 1.5·2^23
    static constexpr unsigned long long kOffset =
        kMagic * (1ull + (1ull << 9) + (1ull << 18) + (1ull << 27) + (1ull << 36) + (kSmall ? 0ull : 1ull << 45));
    static __device__ __forceinline__ void add(unsigned long long &acc, const float D0, const float D1, const float D2,
                                               const float D3, const float D4, const float D5, const float D6) {
        constexpr float M = 12582912.f, up = 0x1p24f, cut = 0x1p15f, back = -0x1p-15f;
        const float b5 = fmaf(fmaf(D6, 0x1p-9f, D5), cut, M);
        const float m4 = fmaf(D4, cut, M), b4 = fmaf(fmaf(m4 - M, back, D4), up, b5);
        const float m3 = fmaf(D3, cut, M), b3 = fmaf(fmaf(m3 - M, back, D3), up, m4);
        const float m2 = fmaf(D2, cut, M), b2 = fmaf(fmaf(m2 - M, back, D2), up, m3);
        const float m1 = fmaf(D1, cut, M), b1 = fmaf(fmaf(m1 - M, back, D1), up, m2);
        long long a = (long long)acc;
        a += (long long)__float_as_int(b4);
        a += (long long)__float_as_int(b3) * (1 << 9);
        a += (long long)__float_as_int(b2) * (1 << 18);
        a += (long long)__float_as_int(b1) * (1 << 27);
        uint32_t hi;
        if (kSmall) {
            hi = (uint32_t)__float_as_int(fmaf(D0, up, m1)) * 16u;
        } else {
            const float m0 = fmaf(D0, cut, M), b0 = fmaf(fmaf(m0 - M, back, D0), up, m1);
            hi = (uint32_t)__float_as_int(b0) * 16u + (uint32_t)__float_as_int(m0) * 8192u;
        }
        acc = (unsigned long long)a + ((unsigned long long)hi << 32);
    }
};

// binary64 V·2^(expo − 1074), rounded to nearest (a tie away from zero)
__device__ __forceinline__ double fixed_to_double(long long V, int expo) {
    const uint32_t sign = (uint32_t)(V >> 32) & 0x80000000u;
    const unsigned long long a = V < 0 ? 0ull - (unsigned long long)V : (unsigned long long)V;
    const uint32_t ahi = (uint32_t)(a >> 32);
    int lz = __clz((int)ahi);
    if (ahi == 0) lz = 32 + __clz((int)(uint32_t)a);  // small against the column's scale: rare
    const int ef = expo + 12 - lz;
    const unsigned long long n = a << (lz & 63);  // leading one at bit 63; V = 0 is set below
    const unsigned long long mant = (n >> 11) + ((uint32_t)(n >> 10) & 1u);
    const unsigned long long bits = mant + ((unsigned long long)((uint32_t)(ef - 1) * 1048576u + sign) << 32);
    double out = __longlong_as_double((long long)bits);
    if ((unsigned)(ef - 1) > 2044u || lz == 64) {  // outside the normal range, or zero: two exact factors
        const int s = expo - 1074, h = s / 2;
        out = V == 0 ? 0.0 : scalbn(scalbn((double)V, h), s - h);
    }
    return out;
}

}  // namespace ss
