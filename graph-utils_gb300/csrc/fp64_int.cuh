// fp64_int.cuh -- pieces of FP64 arithmetic on the integer units.
//
// This part issues two FP64 lanes per clock and SM, 16 clocks for a warp's instruction
// however few of its lanes have work, where an integer instruction takes a quarter clock.
// A division is a dozen FP64 instructions (about 190 clocks of the SM's FP64 unit); the
// one below is some 70 integer ones (about 25 clocks of issue).
#pragma once

#include "device_utils.cuh"

namespace gu {

__host__ __device__ __forceinline__ u64 umul_hi64(u64 a, u64 b)
{
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}

// ma / mb of two mantissas in [2^52, 2^53), as an integer in units of 2^-62, to about
// 2^-61.  r0 is 2^63 / (mb << 11 as 32 upper bits), the reciprocal of mb * 2^-53 in units
// of 2^-31, to 2^-22 relative.  One Newton step gives the reciprocal to 2^-44, the product
// the quotient to 2^-42, and the exact remainder (in 64 bits, wrapping) the rest: the
// remainder form of Markstein (IBM J. Res. Dev. 34, 1990) in fixed point.
__host__ __device__ __forceinline__ u64 mantissa_quotient(u64 ma, u64 mb, unsigned r0)
{
    const u64 ms = mb << 11;
    const u64 T = (ms >> 32) * r0 + (((ms & 0xFFFFFFFFull) * r0) >> 32);  // units of 2^-63, near 1
    const int e = (int)((long long)((1ull << 63) - T) >> 12);             // 1 - m r0, units of 2^-51
    const int half = (int)(r0 >> 1);                                      // r0 in units of 2^-30
    const u64 r1 = ((u64)r0 << 31) + (u64)(((long long)half * e) >> 19);  // units of 2^-62
    const u64 q = umul_hi64(ma << 11, r1) >> 11;                          // ma / mb in units of 2^-51
    const long long rem = (long long)((ma << 51) - q * mb);               // |rem| < 2^62
    return (q << 11) + (u64)(((long long)half * (int)(rem >> 31)) >> 41);
}

// The quotient's bits, rounded to nearest, of two positive doubles (their bits) whose
// exponents and quotient are those of normal numbers; r0 as above, for b's mantissa.
__host__ __device__ __forceinline__ u64 quotient_bits(u64 a, u64 b, unsigned r0)
{
    constexpr u64 M = (1ull << 52) - 1;
    const u64 ma = (a & M) | (M + 1), mb = (b & M) | (M + 1), q = mantissa_quotient(ma, mb, r0);
    const int lt1 = q < (1ull << 62);
    // the mantissa is h or h + 1: which one, the exact remainder from the middle between
    // them tells (in 64 bits, wrapping; below 2^54, and never 0: a quotient of two
    // mantissas of 53 bits does not have 54)
    const u64 h = q >> (lt1 ? 9 : 10);
    const long long past = (long long)((ma << (lt1 ? 54 : 53)) - (2 * h + 1) * mb);
    const u64 m = h + (past > 0);  // [2^52, 2^53]
    return m + ((u64)((int)(a >> 52) - (int)(b >> 52) + 1022 - lt1) << 52);
}

// a / b, rounded to nearest as the division is: for a >= 1 and 1 <= b < 2^64 (so that the
// quotient of a finite a is normal); anything else goes through the division itself.
__device__ __forceinline__ double quotient(double a, double b)
{
    const u64 x = (u64)__double_as_longlong(a), y = (u64)__double_as_longlong(b);
    if (x - (1023ull << 52) >= (1024ull << 52) || y - (1023ull << 52) >= (65ull << 52)) return a / b;
    float g;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(g) : "f"((float)(unsigned)((y >> 21) | 0x80000000u)));
    return __longlong_as_double((long long)quotient_bits(x, y, __float2uint_rz(g * 9223372036854775808.0f)));
}

// (double)x, rounded to nearest even.
__device__ __forceinline__ double u64_to_double(u64 x)
{
    if (!x) return 0.0;
    const int z = __clzll((long long)x);
    const u64 ms = x << z;
    const unsigned rest = (unsigned)ms & 0x7FFu;
    const u64 t = (ms >> 11) + (rest + ((unsigned)(ms >> 11) & 1u) > 0x400u ? 1 : 0);
    return __longlong_as_double((long long)(((u64)(1023 + 63 - 1 - z) << 52) + t));
}

// A sum of positive doubles: acc in units of 2^(e - 1023 - 52 - G), e the largest
// (biased) exponent added, each term rounded to nearest; at most 2^(11 - G) - 1 terms.
template <int G>
struct IntSum {
    u64 acc = 0;
    int e = 0;
    __device__ __forceinline__ void add(double x)
    {
        const u64 b = (u64)__double_as_longlong(x);
        const int ex = (int)(b >> 52);
        u64 m = ((b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << G;
        const int up = max(ex - e, 0), down = max(e - ex, 0);
        acc = up < 64 ? acc >> up : 0ull;  // (the dropped bits: less than a unit, once per new largest term)
        e = max(e, ex);
        m = down < 60 ? (m + ((1ull << down) >> 1)) >> down : 0ull;
        acc += m;
    }
    // what add() may be given: zero and normal numbers, here those that add something
    __device__ __forceinline__ static bool takes(double x)
    {
        const unsigned ex = (unsigned)((u64)__double_as_longlong(x) >> 52);
        return ex - 1u < 2046u;
    }
    __device__ __forceinline__ double value() const { return acc ? scalbn((double)acc, e - 1023 - 52 - G) : 0.0; }
};
// The sum of the 32 lanes' sums (each below 2^63): 96 bits in units 2^24 times finer than
// those of the largest exponent, rounded once.
template <int G>
__device__ __forceinline__ double warp_total(const IntSum<G> &s)
{
    const int em = __reduce_max_sync(FULL_MASK, s.e), d = em - s.e;
    u64 hi = d < 56 ? s.acc >> (d + 8) : 0ull;
    unsigned lo = d <= 24 ? (unsigned)(s.acc << (24 - d)) : d < 88 ? (unsigned)(s.acc >> (d - 24)) : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const u64 h2 = __shfl_xor_sync(FULL_MASK, hi, o);
        const unsigned l2 = __shfl_xor_sync(FULL_MASK, lo, o), sum = lo + l2;
        hi += h2 + (sum < l2);
        lo = sum;
    }
    if (!hi) return 0.0;  // nothing added: a term leaves 2^(44 + G) here
    const int z = __clzll((long long)hi);  // 4 .. 19 - G
    const u64 ms = hi << z | lo >> (32 - z) | (lo << z ? 1u : 0u);
    const int k = em - 1023 - 52 - G - 24 + 32 - z;
    const double x = u64_to_double(ms);  // in [2^63, 2^64]
    if (k <= -1086 || k >= 960) return scalbn(x, k);
    return __longlong_as_double(__double_as_longlong(x) + ((long long)k << 52));
}

}  // namespace gu
