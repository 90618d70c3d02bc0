/* Compares the quotients of cuphu_b200/csrc/quotient.cuh with the division operator.  Prints per
 * function the number of pairs and of differences. */
#include "quotient.cuh"

#include <stdio.h>

using namespace cuphu;

static uint64_t g_state = 0x9e3779b97f4a7c15ull;
static uint64_t next()
{
    g_state ^= g_state << 13;
    g_state ^= g_state >> 7;
    g_state ^= g_state << 17;
    return g_state;
}
/* a significand: random, all ones, zero, or near the two */
static uint64_t significand()
{
    const uint64_t ones = (1ull << 52) - 1;
    switch (next() % 8) {
    case 0: return ones;
    case 1: return 0;
    case 2: return ones - next() % 4;
    case 3: return next() % 4;
    default: return next() & ones;
    }
}
static double number(int elo, int ehi)   /* biased exponents */
{
    return bits_double(((uint64_t)(elo + (int)(next() % (uint64_t)(ehi - elo + 1))) << 52) |
                       significand());
}
static bool same(double a, double b)
{
    return (isnan(a) && isnan(b)) || double_bits(a) == double_bits(b);
}

int main()
{
    long n[4] = {0, 0, 0, 0}, bad[4] = {0, 0, 0, 0};
    auto take = [&](int k, double got, double want) {
        ++n[k];
        if (!same(got, want)) ++bad[k];
    };
    for (long i = 0; i < 3000000; ++i) {
        /* the scalars of a solve, then any exponents, then results at both ends of the range */
        double a = number(1000, 1100), b = number(1000, 1100);
        take(0, quotient_any(a, b), a / b);
        a = number(0, 2047), b = number(0, 2047);
        take(1, quotient_any(a, b), a / b);
        a = bits_double(double_bits(a) ^ (next() << 63));
        take(1, quotient_any(a, b), a / b);
        const int e = 1 + (int)(next() % 1100);
        a = number(e, e), b = number(e + 1015 + (int)(next() % 70) < 2046 ? e + 1015 : 2046, 2046);
        take(2, quotient_any(a, b), a / b);
        take(2, quotient_any(b, a), b / a);
        /* a pixel's r / diag from the rounded reciprocal, over the range of its comment */
        double r = bits_double(double_bits(number(123, 1922)) ^ (next() << 63)), d = number(923, 1122);
        if (i % 64 == 0) r = 0.0;
        if (!res_odd(r)) take(3, quotient(r, d, 1.0 / d), r / d);
    }
    const double edge[] = {0.0, 1.0, bits_double(1), bits_double((1ull << 52) - 1),
                           bits_double(1ull << 52), bits_double((0x7ffull << 52) - 1),
                           bits_double(0x7ffull << 52), bits_double(0x7ff8ull << 48),
                           ldexp(1.0, 600), ldexp(1.0, -600), ldexp(1.0, 900), ldexp(1.0, -900)};
    for (double a : edge)
        for (double b : edge) {
            take(1, quotient_any(a, b), a / b);
            take(1, quotient_any(-a, b), -a / b);
        }
    const char *name[4] = {"scalars", "any", "ends", "pixels"};
    for (int k = 0; k < 4; ++k) printf("%s %ld %ld\n", name[k], n[k], bad[k]);
    return 0;
}
