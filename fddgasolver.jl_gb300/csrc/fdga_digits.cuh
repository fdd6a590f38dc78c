// fdga_digits.cuh -- FP64 values as fixed-point integers and back, on the integer pipes (shared by the
// digit-sliced K3 contractions, fdga_k3_oz.cu and fdga_k3_mma.cu).
#pragma once
#include "fdga_device.cuh"

namespace fdga {

// the exponent field of an FP64 value
__device__ __forceinline__ int efield(double v) {
    return (int)(((unsigned long long)__double_as_longlong(v) >> 52) & 0x7ffull);
}
// the larger exponent field of the two parts of a complex number: both |x|, |y| < 2^(E - 1022)
// (zero and subnormal parts included, with E = 0)
__device__ __forceinline__ int cexpo(cplx v) { return max(efield(v.x), efield(v.y)); }
// x · 2^e for an integer |x| < 2^53 (exact), built from its bits on the integer pipes; 0 below the
// normal range
__device__ __forceinline__ double i2d_scaled(long long x, int e) {
    if (x == 0) return 0.0;
    const unsigned long long sg = x < 0 ? (1ull << 63) : 0ull;
    const unsigned long long u = x < 0 ? (unsigned long long)(-x) : (unsigned long long)x;
    const int p = 63 - __clzll((long long)u);  // 2^p ≤ u < 2^(p+1), p ≤ 52
    const int ef = p + e + 1023;
    if (ef <= 0) return 0.0;
    if (ef >= 2047) return __longlong_as_double((long long)(sg | 0x7FF0000000000000ull));
    const unsigned long long mant = (u << (52 - p)) & 0xFFFFFFFFFFFFFull;
    return __longlong_as_double((long long)(sg | ((unsigned long long)ef << 52) | mant));
}

// An FP64 value as S balanced base-256 digits relative to a bound 2^(F-1022) > |v|: Y = v 2^(8S-2+1022-F)
// rounded to an integer (0 for zero and subnormal v), |Y| ≤ 2^(8S-2); adding 0x80 to every byte of Y makes
// byte k < S, less 128, the digit of weight 256^k, in [-128, 127].  S = 8: 62 fractional bits, exact for every
// v within 2^9 of the bound.
template <int S>
__device__ __forceinline__ long long fixed_digits(double v, int F) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int ev = (int)((b >> 52) & 0x7ffull);
    const int rs = F - ev - (8 * S - 55);
    if (ev == 0 || rs >= 55) return 0;
    const unsigned long long mant = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const long long y = (long long)(rs < 0 ? mant << (-rs) : (rs == 0 ? mant : (mant + (1ull << (rs - 1))) >> rs));
    return (long long)b < 0 ? -y : y;
}
constexpr unsigned long long DIGIT_BIAS = 0x8080808080808080ull;
// digit k (from the least significant) of two biased integers as a pair of FP16 numbers (exact: 0x6400 | byte
// is 1024 + byte, less 1152)
__device__ __forceinline__ uint32_t digit_pair(unsigned long long a, unsigned long long b, int k) {
    const uint32_t x = k < 4 ? (uint32_t)a : (uint32_t)(a >> 32), y = k < 4 ? (uint32_t)b : (uint32_t)(b >> 32);
    const uint32_t i = (uint32_t)(k & 3);
    const uint32_t u = (__byte_perm(x, y, i | ((4u + i) << 8)) & 0x00ff00ffu) | 0x64006400u;
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(u), "r"(0x64806480u));  // 0x6480 = 1152
    return r;
}
// the product of two such numbers from its S integer diagonals acc_g = Σ_{s+t=g} (digit s)·(digit t) (from
// the most significant; |acc_g| ≤ 2^25) and the two bounds: Σ_g 256^(2(S-1)-g) acc_g 2^(F_A + F_M - 2044 -
// 2(8S-2)), joined exactly in two 64-bit integers and one FP64 addition
template <int S>
__device__ __forceinline__ double join_digits(const float (&acc)[S], int fsum) {
    const int E = fsum - 2044 - 2 * (8 * S - 2);
    long long hi = 0, lo = 0;
#pragma unroll
    for (int g = 0; g < S; ++g) {
        const long long v = (long long)__float2int_rn(acc[g]);
        if (g < 4) hi = hi * 256 + v;
        else lo = lo * 256 + v;
    }
    return i2d_scaled(hi, E + 8 * (2 * (S - 1) - 3)) + i2d_scaled(lo, E + 8 * (S - 1));
}

}  // namespace fdga
