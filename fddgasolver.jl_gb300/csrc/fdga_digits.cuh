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

}  // namespace fdga
