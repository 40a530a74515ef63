// gw_math64.cuh -- FP64 exp and log for the global step's lane program, in 64-bit integer arithmetic.
//
// On GB300 a warp's FP64 instruction occupies its SM sub-partition's FP64 unit for ~64 cycles, with
// or without instruction-level parallelism; a dependent integer instruction takes 4 to 5.  So both
// functions run in fixed point (table reduction and Taylor polynomials, as in Tang's table-driven
// methods, ACM TOMS 15(2) 1989 and 16(4) 1990, but on integers):
//   exp: x / ln2 = n + f, from the 128-bit product of x's significand with 1/ln2 (64 bits); f = j/256 + t,
//        2^t - 1 its degree-5 Taylor polynomial with 64-bit products, the last two coefficients in
//        32 bits (their terms are below 2^-30 of the sum); exp(x) = 2^n 2^(j/256) 2^t.
//   log: x = 2^e m, c_j >= 2^16 / (1 + j/256) from the leading 8 fraction bits, u = m c_j / 2^16 - 1
//        exactly (0 <= u < 2^-7.9), log(x) = e ln2 - log(c_j / 2^16) + log1p(u), log1p by its degree-7 Taylor
//        polynomial, summed with 64 fractional bits and rounded once.
// Error against 64-bit-significand libm over 2e7 arguments each: exp 0.513 ulp for |x| < 50 and 0.62 for
// |x| < 700 (the FP64 form they replace: 0.81), log 0.51 away from 1 (1.25).  Latency of one call by a
// warp, measured: exp 370 cycles (882 in FP64), log 580 (989).
// Inputs outside the reduced ranges (|x| >= 700 for exp; non-positive, non-normal, non-finite
// or within 2^-5 of 1 for log) take CUDA's exp / log.  Tables (generated by gen_math_tables.py from
// 80-digit decimal arithmetic) are copied to shared memory once per launch.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "gw_math_tables.h"

namespace gw {
namespace math64 {

struct LogEntry {
    unsigned long long c;  // c_j
    unsigned long long l;  // -log(c_j / 2^16)
};
struct Tables {
    unsigned long long e2[256];
    LogEntry lg[256];
};

static __constant__ unsigned long long c_exp2_table[256] = GW_EXP2_TABLE;
static __constant__ unsigned long long c_log_table[256][2] = GW_LOG_TABLE;

// Copies the tables to shared memory; threads tid = 0 .. n-1 of the caller take part.
__device__ __forceinline__ void load_tables(Tables &T, int tid, int n) {
    for (int i = tid; i < 256; i += n) {
        T.e2[i] = c_exp2_table[i];
        T.lg[i].c = c_log_table[i][0];
        T.lg[i].l = c_log_table[i][1];
    }
}

// The high word of a b without the product of the low halves: up to 2 less (__umul64hi's carries take
// 60 cycles, this 25).
__device__ __forceinline__ unsigned long long mulhi(unsigned long long a, unsigned long long b) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    return (unsigned long long)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

// 64-bit significand r (leading bit 63) times 2^(e - 63), rounded to double (e + 1022 the biased
// exponent less one: the significand's own leading bit, and a carry out of it, complete it).
__device__ __forceinline__ unsigned long long pack(unsigned long long r, int e) {
    return (r >> 11) + ((r >> 10) & 1ull) + ((unsigned long long)(uint32_t)(e + 1022) << 52);
}

__device__ __forceinline__ double exp(double x, const Tables &T) {
    const uint32_t xh = (uint32_t)__double2hiint(x), xl = (uint32_t)__double2loint(x);
    const uint32_t ah = xh & 0x7FFFFFFFu;
    if (ah >= 0x4085E000u) return ::exp(x);  // |x| >= 700, inf, NaN
    const unsigned long long M =
        ((unsigned long long)(((ah & 0xFFFFFu) << 11) | 0x80000000u | (xl >> 21)) << 32) | (xl << 11);
    const unsigned long long ph = __umul64hi(M, kLog2e63), pl = M * kLog2e63;
    // |x| / ln2 = (ph : pl) 2^-(64 + k): the integer part n, and the fraction f of 64 bits
    const int k = 1085 - (int)(ah >> 20);
    unsigned long long f;
    int n = 0;
    if (k < 64) {  // |x| >= 1/2
        f = (ph << (64 - k)) | (pl >> k);
        n = (int)(ph >> k);
    } else {
        f = k < 128 ? ph >> (k - 64) : 0ull;
    }
    if ((int)xh < 0) {
        n = -n - (f != 0ull ? 1 : 0);
        f = 0ull - f;
    }
    const unsigned long long e2 = T.e2[f >> 56], u = f << 8;
    const uint32_t uh = (uint32_t)(u >> 32);
    const uint32_t a4 = kExp4 + (__umulhi(uh, kExp5) >> 8);
    const unsigned long long a3 = kExp3 + (((unsigned long long)uh * a4) >> 8);
    const unsigned long long a2 = kExp2 + (mulhi(u, a3) >> 8);
    const unsigned long long a1 = kExp1 + (mulhi(u, a2) >> 8);
    const unsigned long long p = mulhi(u, a1);  // (2^t - 1) 2^72
    return __longlong_as_double((long long)pack(e2 + (mulhi(e2, p) >> 8), n));
}

__device__ __forceinline__ double log(double x, const Tables &T) {
    const long long b = __double_as_longlong(x);
    // positive normal finite and not within 2^-5 of 1 (there log(x) is small and the sum would cancel)
    const bool normal = (unsigned long long)(b - 0x0010000000000000ll) < 0x7FE0000000000000ull;
    const bool near1 = (unsigned long long)(b - 0x3FEF000000000000ll) < 0x0001800000000000ull;
    if (!normal || near1) return ::log(x);
    const uint32_t hi = (uint32_t)((unsigned long long)b >> 32);
    const LogEntry t = T.lg[(hi >> 12) & 0xFFu];
    const unsigned long long m = ((unsigned long long)b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
    const unsigned long long U = (m * t.c) << 3;  // u 2^71: the product less 2^68, modulo 2^64
    const uint32_t uh = (uint32_t)(U >> 32);
    const uint32_t b6 = kLog6 - (__umulhi(uh, kLog7) >> 7);
    const uint32_t b5 = kLog5 - (__umulhi(uh, b6) >> 7);
    const uint32_t b4 = kLog4 - (__umulhi(uh, b5) >> 7);
    const unsigned long long b3 = kLog3 - (((unsigned long long)uh * b4) >> 7);
    const unsigned long long b2 = kLog2 - (mulhi(U, b3) >> 7);
    const unsigned long long b1 = 0ull - (mulhi(U, b2) >> 7);  // (1 - u b2) 2^64, modulo 2^64
    const unsigned long long q = ((b1 ? mulhi(U, b1) : U) + 64ull) >> 7;  // log1p(u) 2^64
    // e ln2 + table + q in 128 bits, e biased to be positive
    const uint32_t eb = (hi >> 20) + 1025u;  // e + 2048
    const unsigned long long p0 = (unsigned long long)eb * (uint32_t)kLn2;
    const unsigned long long p1 = (unsigned long long)eb * (uint32_t)(kLn2 >> 32) + (p0 >> 32);
    unsigned long long vl = (p1 << 32) | (uint32_t)p0, vh = p1 >> 32;
    unsigned long long w = vl - kLn2BiasLo;
    vh = vh - kLn2BiasHi - (vl < kLn2BiasLo ? 1ull : 0ull);
    vl = w + t.l;
    vh += vl < w ? 1ull : 0ull;
    w = vl + q;
    vh += w < vl ? 1ull : 0ull;
    vl = w;
    const bool neg = (long long)vh < 0;
    if (neg) {
        vh = ~vh + (vl == 0ull ? 1ull : 0ull);
        vl = 0ull - vl;
    }
    // |log(x)| = (vh : vl) 2^-64 with vh < 2^10, and at least 2^-5: leading bit to 63
    const uint32_t v32 = (uint32_t)vh;
    const int s = v32 ? 32 - __clz((int)v32) : -__clz((int)(vl >> 32));
    const unsigned long long r = v32 ? (vh << (64 - s)) | (vl >> s) : vl << -s;
    const unsigned long long o = pack(r, s - 1);
    return __longlong_as_double((long long)(neg ? o | 0x8000000000000000ull : o));
}

}  // namespace math64
}  // namespace gw
