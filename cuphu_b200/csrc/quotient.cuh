/*
 * quotient.cuh -- FP64 quotients without the division operator, for the
 * iterations of the on-chip FP64 solver (resident_fp64.cu, which names the
 * source of the correction steps): the call that the operator can make would
 * cost the loop its registers.  Compiles for the host as well, where
 * tests/test_quotients.py compares them with the operator.
 */
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define CUPHU_QUOTIENT __host__ __device__ __forceinline__
#else
#define CUPHU_QUOTIENT static inline
#endif

namespace cuphu {

CUPHU_QUOTIENT uint64_t double_bits(double v)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    memcpy(&u, &v, sizeof u);
    return u;
#endif
}
CUPHU_QUOTIENT double bits_double(uint64_t u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v;
    memcpy(&v, &u, sizeof v);
    return v;
#endif
}

/* 1 / b to some 20 bits, b a normal number */
CUPHU_QUOTIENT double reciprocal_seed(double b)
{
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
#else
    int e;
    const float m = (float)frexp(b, &e);
    return ldexp((double)(1.0f / m), -e);
#endif
}

/* r / d from y = RN(1/d).  The correction steps are exact where nothing
 * underflows or overflows: for a residual that is zero or in [2^-900, 2^900]
 * (res_odd tests the rest) and a diagonal in [2^-100, 2^100] (y = 0 marks the
 * rest).  A block that meets another value forms its quotients with IEEE
 * divisions, in functions of their own (slow_fold, slow_update). */
CUPHU_QUOTIENT double quotient(double r, double d, double y)
{
    const double q0 = r * y;
    const double q1 = fma(fma(-q0, d, r), y, q0);
    return fma(fma(-q1, d, r), y, q1);
}
CUPHU_QUOTIENT bool res_odd(double r)
{
    const unsigned e = ((unsigned)(double_bits(r) >> 32) & 0x7fffffffu) - (123u << 20);
    return e > (1800u << 20) && r != 0.0;
}

/* a / b by long division, rounded to nearest even: zeros, infinities, NaN,
 * subnormal operands and results, overflow */
CUPHU_QUOTIENT double quotient_digits(double a, double b)
{
    constexpr uint64_t kInf = 0x7ffull << 52, kLead = 1ull << 52, kSign = 1ull << 63;
    uint64_t ma = double_bits(a), mb = double_bits(b);
    const uint64_t sign = (ma ^ mb) & kSign;
    ma &= ~kSign;
    mb &= ~kSign;
    if (ma > kInf || mb > kInf || (ma == mb && (ma == 0 || ma == kInf)))
        return bits_double(kInf | (kLead >> 1));
    if (ma == kInf || mb == 0) return bits_double(sign | kInf);
    if (mb == kInf || ma == 0) return bits_double(sign);
    /* significands with the leading bit, exponents */
    int ea = (int)(ma >> 52), eb = (int)(mb >> 52);
    ma = ea ? (ma & (kLead - 1)) | kLead : ma;
    mb = eb ? (mb & (kLead - 1)) | kLead : mb;
    ea += ea == 0;
    eb += eb == 0;
    for (; ma < kLead; --ea) ma <<= 1;
    for (; mb < kLead; --eb) mb <<= 1;
    int e = ea - eb + 1023;
    if (ma < mb) {
        ma <<= 1;
        --e;
    }
    if (e >= 2047) return bits_double(sign | kInf);
    /* 55 digits, the last one also set by a remainder */
    uint64_t q = 0;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (int k = 0; k < 55; ++k) {
        q <<= 1;
        if (ma >= mb) {
            ma -= mb;
            q |= 1;
        }
        ma <<= 1;
    }
    q |= ma != 0;
    /* two digits too many, more of them where the result is subnormal (a shift
     * of 58 leaves nothing, and what it drops is less than a half) */
    const int sh = e > 0 ? 2 : e < -54 ? 58 : 3 - e;
    const uint64_t rest = q & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    uint64_t m = q >> sh;
    m += rest > half || (rest == half && (m & 1));
    return bits_double(sign | (m + ((uint64_t)(e > 0 ? e - 1 : 0) << 52)));
}

/* a / b, the operator's value for every pair of operands (any NaN for a NaN).
 * Operands in [2^-400, 2^400]: the reciprocal by Newton steps from the
 * hardware's approximation, which is the correctly rounded one unless the
 * divisor's significand is all ones (there it is the next number above a power
 * of two), then Markstein's correction steps.  All others, which the scalars
 * of a solve meet only when it over- or underflows, by digits. */
CUPHU_QUOTIENT double quotient_any(double a, double b)
{
    const uint64_t ua = double_bits(a), ub = double_bits(b);
    const unsigned ea = (unsigned)(ua >> 52) - 623u, eb = (unsigned)(ub >> 52) - 623u;
    const bool odd = ea > 800u || eb > 800u;
    double y = reciprocal_seed(b);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = 0; k < 3; ++k) y = fma(y, fma(-b, y, 1.0), y);
    if (((ub + 1) & ((1ull << 52) - 1)) == 0) y = bits_double(((2045ull - (ub >> 52)) << 52) | 1);
    const double q = quotient(a, b, y);
    return __builtin_expect(odd, 0) ? quotient_digits(a, b) : q;   /* off the usual path's way */
}

}  // namespace cuphu
