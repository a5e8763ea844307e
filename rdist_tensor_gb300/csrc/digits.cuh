// FP64 values as balanced base-256 digits: a digit is exact in bf16, a product
// of two and sums of up to 2^10 of them are exact in the tensor core's FP32
// accumulators, so products of digit slices are exact integer arithmetic
// (Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix
// multiplication", 2012, with digits of eight bits).
#pragma once
#include "common.cuh"
#include "umma.cuh"

namespace exafac {

// kind::f16: D FP32, A and B bf16, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
// Biased exponent of |v| (0 for zero and subnormals, 2047 for inf and nan).
__device__ __forceinline__ int bexp(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// v 2^(1028 - emax), below 2^6 where |v| < 2^(emax - 1022), as an integer in
// units of 2^-56 (toward zero).
__device__ __forceinline__ long long fix56(double v, int emax) {
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7ff);
    unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
    if (e) m |= 1ull << 52;
    const int s = max(max(emax, 1) - max(e, 1), 0);
    m = s > 63 ? 0ull : (m << 9) >> s;
    return b < 0 ? -(long long)m : (long long)m;
}

// (byte idx of t - 128) 2^-8w as a float (exact).
template <int W>
__device__ __forceinline__ float digit_f(uint32_t t, uint32_t idx) {
    constexpr float sc = W == 0 ? 1.0f : W == 1 ? 0x1p-8f : W == 2 ? 0x1p-16f : W == 3 ? 0x1p-24f
                         : W == 4 ? 0x1p-32f : W == 5 ? 0x1p-40f : W == 6 ? 0x1p-48f : 0x1p-56f;
    return fmaf(__uint_as_float(__byte_perm(t, 0x4B000000u, 0x7440u | idx)), sc, -8388736.0f * sc);
}
__device__ __forceinline__ float lead_f(int d) {  // |d| <= 128 as a float
    return __int_as_float(0x4B400000 + d) - 12582912.0f;
}
// two exact bf16 values, given as floats, packed (lo in the low half)
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632u);
}

}  // namespace exafac
