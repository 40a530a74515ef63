// gw_div64.cuh -- correctly rounded FP64 division and square root on the integer and FP32 pipes.
//
// GB300's FP64 pipe takes one warp instruction per ~64 cycles per SM sub-partition; a division through
// it is about ten of them.  This one is long division on the 53-bit significands: a reciprocal
// estimate of the divisor in FP32 (relative error within 2^-21.5 with the truncation of its argument)
// gives the quotient in three signed digits of 20, 16 and 16 bits, each followed by the exact remainder
// in 64-bit integer arithmetic (modulo 2^64; the true remainder stays below 1.5, 0.6 and 0.6 divisors),
// and the last remainder rounds the quotient to nearest.  A quotient of 53-bit significands is never
// halfway between two 53-bit numbers, so the result is the IEEE one wherever both operands and the
// quotient are normal numbers; everything else takes the hardware's division.
//
// What it is bound by: ~60 integer and FP32 instructions.  Measured on GB300, dependent divisions by one
// warp: 235 cycles each (a / b: 600); with 16 warps per SM ~55 cycles of a sub-partition each (565).
//
// The square root goes the same way: the root's leading 20 bits from an FP32 reciprocal square root
// (relative error within 2^-21 with its argument's truncation), two signed digits of 16 bits from the
// exact remainder x - s^2, the last remainder rounding to nearest (the root of a 53-bit significand is
// never halfway either).  ~55 instructions.
#pragma once

#include <cmath>
#include <cstdint>

namespace gw {

#if defined(__CUDA_ARCH__)

// Operands or quotients outside the normal range (zero, subnormal, infinite, NaN, near over- and
// underflow): out of line, so that the common path carries no copy of it.
static __device__ __noinline__ double div_special(double a, double b) { return a / b; }

__device__ __forceinline__ float rcp_estimate(float y) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    return r;
}

__device__ __forceinline__ double div_rn(double a, double b) {
    const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
    const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
    const uint32_t ea = (ah >> 20) & 0x7FFu, eb = (bh >> 20) & 0x7FFu;
    const int e = (int)ea - (int)eb;
    if (ea - 1u >= 2046u || eb - 1u >= 2046u || (uint32_t)(e + 1020) >= 2040u) return div_special(a, b);
    const uint32_t Bh = (bh & 0xFFFFFu) | 0x100000u, Ah = (ah & 0xFFFFFu) | 0x100000u;
    // dividend significand doubled where it is the smaller, so that the quotient lies in [1, 2)
    const bool lt = Ah < Bh || (Ah == Bh && al < bl);
    const uint32_t s = lt ? 1u : 0u;
    const float y = rcp_estimate(__uint_as_float((__funnelshift_l(bl, bh, 3) & 0x7FFFFFu) | 0x3F800000u));
    const float x = __uint_as_float(((__funnelshift_l(al, ah, 3) & 0x7FFFFFu) | 0x3F800000u) + (s << 23));
    // divisor as bl (signed) + 2^32 Bs, for signed 32 x 32 -> 64 products
    const int bs = (int)bl, Bs = (int)(Bh + (bl >> 31));
    const float y2 = y * 0.0625f;
    // A digit is the low bits of (estimate + 1.5 * 2^23); n1, n2, n3 are the digits negated.
    const int n1 = (int)(0x4B400000u - __float_as_uint(__fmaf_rn(x, y * 1048576.f, 12582912.f)));
    const uint32_t rs = 20u + s;
    unsigned long long r = ((unsigned long long)__funnelshift_l(al, Ah, rs) << 32) | (al << rs);
    r += (unsigned long long)((long long)n1 * (long long)bs) + ((unsigned long long)(uint32_t)(n1 * Bs) << 32);
    float f = __uint_as_float(0x4B400000u + (uint32_t)(r >> 32)) - 12582912.f;
    const int n2 = (int)(0x4B400000u - __float_as_uint(__fmaf_rn(f, y2, 12582912.f)));
    r = (r << 16) + (unsigned long long)((long long)n2 * (long long)bs) + ((unsigned long long)(uint32_t)(n2 * Bs) << 32);
    f = __uint_as_float(0x4B400000u + (uint32_t)(r >> 32)) - 12582912.f;
    const int n3 = (int)(0x4B400000u - __float_as_uint(__fmaf_rn(f, y2, 12582912.f)));
    r = (r << 16) + (unsigned long long)((long long)n3 * (long long)bs) + ((unsigned long long)(uint32_t)(n3 * Bs) << 32);
    // quotient significand with its leading bit at 2^52, the remainder's sign rounding it
    const long long B = (long long)(((unsigned long long)Bh << 32) | bl), d = (long long)(r << 1);
    const int adj = (d > B ? 1 : 0) - (d < -B ? 1 : 0);
    const long long lo = (long long)n2 * 65536ll + (long long)(n3 - adj);
    const unsigned long long N = ((unsigned long long)(uint32_t)(-n1) << 32) - (unsigned long long)lo;
    const uint32_t top = ((uint32_t)(e - (int)s + 1022) << 20) + ((ah ^ bh) & 0x80000000u);
    return __longlong_as_double((long long)(N + ((unsigned long long)top << 32)));
}

// Negative, zero, subnormal, infinite or NaN arguments.
static __device__ __noinline__ double sqrt_special(double x) { return sqrt(x); }

__device__ __forceinline__ double sqrt_rn(double x) {
    const uint32_t xh = (uint32_t)__double2hiint(x), xl = (uint32_t)__double2loint(x);
    const uint32_t ex = xh >> 20;  // with the sign, so that a negative x is out of range
    if (ex - 1u >= 2046u) return sqrt_special(x);
    const uint32_t odd = (ex & 1u) ^ 1u;  // an odd exponent of x doubles the significand
    const uint32_t Xh = (xh & 0xFFFFFu) | 0x100000u;
    const float v = __uint_as_float(((__funnelshift_l(xl, xh, 3) & 0x7FFFFFu) | 0x3F800000u) + (odd << 23));
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(v));
    const float y4 = y * 0.0625f;
    // root s1 in units of 2^-20, remainder in units of 2^-52
    const int s1 = __float_as_int(__fmaf_rn(v * y, 1048576.f, 12582912.f)) - 0x4B400000;
    unsigned long long r = ((unsigned long long)__funnelshift_l(xl, Xh, odd) << 32) | (xl << odd);
    r -= (unsigned long long)((long long)s1 * (long long)s1) << 12;
    float f = __int_as_float(0x4B400000 + (int)((long long)r >> 13)) - 12582912.f;
    const int d2 = __float_as_int(__fmaf_rn(f, y4, 12582912.f)) - 0x4B400000;
    r = (r << 20) - ((unsigned long long)((long long)s1 * (long long)d2) << 17) -
        (unsigned long long)((long long)d2 * (long long)d2);  // units of 2^-72
    f = __int_as_float(0x4B400000 + (int)((long long)r >> 17)) - 12582912.f;
    const int d3 = __float_as_int(__fmaf_rn(f, y4, 12582912.f)) - 0x4B400000;
    const long long s2 = ((long long)s1 << 16) + d2;  // units of 2^-36
    r = (r << 32) - (((unsigned long long)s2 * (unsigned long long)(long long)d3) << 17) -
        (unsigned long long)((long long)d3 * (long long)d3);  // units of 2^-104
    const long long S = (s2 << 16) + d3, R = (long long)r;
    const long long root = S + (R > S ? 1 : 0) - (R <= -S ? 1 : 0);
    return __longlong_as_double(root + ((long long)(((ex + 1023u - odd) >> 1) - 1u) << 52));
}

#else

inline double div_rn(double a, double b) { return a / b; }
inline double sqrt_rn(double x) { return std::sqrt(x); }

#endif

}  // namespace gw
