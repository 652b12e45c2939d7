// exact_int_check.cpp -- products, small-constant products, quotients and
// square roots of exact_int.cuh against the host's IEEE arithmetic, bit for
// bit, on n seeded operand pairs: every exponent, short and all-ones
// significands, products and quotients near rounding midpoints, equal and
// neighbouring operands, squares and their neighbours.  Prints the
// mismatches of each; exit code 1 if there is any.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "exact_int.cuh"

using namespace cfd::xi;

static uint64_t bits(double x)
{
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return u;
}

static double from(uint64_t u)
{
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}

static bool same(double a, double b) { return (a != a && b != b) || bits(a) == bits(b); }

template <int C, int K>
static long small_bad(double x)
{
    uint32_t h, l;
    if (small_words<C, K>(x, h, l)) return 0;   // outside the plain case: the caller multiplies
    volatile double r = x * std::ldexp((double)C, K);
    return bits(r) != (((uint64_t)h << 32) | l);
}

static long root_bad(double x)
{
    volatile double r = std::sqrt(x);
    return !same(root(x), r);
}

int main(int argc, char **argv)
{
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    std::mt19937_64 g(argc > 2 ? std::atol(argv[2]) : 1);
    long mul_n_bad = 0, small_n_bad = 0, div_bad = 0, sqrt_bad = 0;
    for (long i = 0; i < n; ++i) {
        uint64_t a = g(), b = g();
        const int kind = (int)(i % 8);
        if (kind == 1) {
            a &= ~((1ull << (g() % 52)) - 1);
            b &= ~((1ull << (g() % 52)) - 1);
        } else if (kind == 2) {
            a |= (1ull << (g() % 50)) - 1;
            b |= (1ull << (g() % 50)) - 1;
        } else if (kind == 3) {
            a = (a & ~((1ull << 26) - 1)) + (g() % 3) - 1;
            b &= ~((1ull << 25) - 1);
        } else if (kind == 4) {
            b = a + (g() % 7) - 3;
        } else if (kind == 5) {
            a = (a & ~0xfffffffffffffull) | (g() % 5);
        } else if (kind == 6) {
            b = (b & ~0xfffffffffffffull) | (g() % 5) | (g() % 2 ? 0xffffffffffff0ull : 0);
        } else if (kind == 7) {   // x / b next to a midpoint
            const uint64_t q = (g() >> 11) | (1ull << 52);
            const double d = std::ldexp((double)((b >> 12) | (1ull << 52)), -52);
            a = bits((double)(((long double)q + 0.5L) * d));
            b = bits(d);
        }
        if (kind >= 1 && kind <= 6) {   // everyday exponents
            a = (a & 0x800fffffffffffffull) | ((uint64_t)(900 + g() % 300) << 52);
            b = (b & 0x800fffffffffffffull) | ((uint64_t)(900 + g() % 300) << 52);
        }
        const double x = from(a), y = from(b);
        volatile double p = x * y, q = x / y;
        mul_n_bad += !same(mul(x, y), p);
        div_bad += !same(divide(x, y), q);
        small_n_bad += small_bad<3, 0>(x) + small_bad<3, -3>(x) + small_bad<5, -2>(x) + small_bad<5, 0>(x)
                       + small_bad<15, -3>(x) + small_bad<17, 1>(x) + small_bad<39, 0>(x) + small_bad<63, 8>(x);
        sqrt_bad += root_bad(std::fabs(x)) + root_bad(x);
        const double r = std::ldexp((double)((a >> 12) | (1ull << 51)), -51);
        for (int z = -2; z <= 2; ++z) sqrt_bad += root_bad(from(bits(r * r) + z));
    }
    std::printf("%ld pairs: %ld product mismatches, %ld small-constant mismatches, %ld quotient mismatches, "
                "%ld root mismatches\n",
                n, mul_n_bad, small_n_bad, div_bad, sqrt_bad);
    return mul_n_bad || small_n_bad || div_bad || sqrt_bad;
}
