// seed_bound_check.cpp -- the quotients and square roots of exact_int.cuh
// from seeds as far from the exact value as the device's approximations may
// be (PTX: rcp.approx.f32 within 2^-23 for operands in [1, 2), two units of the
// seed's last place; rsqrt.approx.f32 within 2^-22.9 of the value), in either direction, for every significand a seed is formed of: 2^23 of the
// reciprocal, 2^24 of the reciprocal root (both parities of the exponent).
// Prints the results whose bits differ from the host's operations; exit code
// 1 if there is any.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

static int g_ulps = 0;   // the seeds' error in units of their last place

// The value `ulps` last places of [1/2, 1) from the nearest to x, stepping
// over 1/2 and 1 as the device's roundings would.
static float off(double x)
{
    float f = (float)x;
    for (int k = 0; k < (g_ulps < 0 ? -g_ulps : g_ulps); ++k) f = std::nextafterf(f, g_ulps < 0 ? 0.0f : 2.0f);
    return f;
}
#define CFD_XI_HOST_RCP(m) off(1.0 / (double)(m))
#define CFD_XI_HOST_RSQRT(m) off(1.0 / std::sqrt((double)(m)))
#include "exact_int.cuh"

using namespace cfd::xi;

static double from(uint64_t u)
{
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}

static bool same(double a, double b) { return std::memcmp(&a, &b, 8) == 0; }

int main()
{
    long total = 0;
    for (int u = -2; u <= 2; ++u) {
        g_ulps = u;
        long div_bad = 0, root_bad = 0;
        uint64_t s = 88172645463325252ull + u;
        for (uint64_t m = 0; m < (1ull << 23); ++m) {
            s ^= s << 13;
            s ^= s >> 7;
            s ^= s << 17;
            const uint64_t low = m % 3 == 0 ? 0 : (m % 3 == 1 ? 0x1fffffffull : (s & 0x1fffffffull));
            const uint64_t B = (m << 29) | low;
            const double b = from((1023ull << 52) | B), x = from((1023ull << 52) | (s >> 12));
            volatile double q = x / b, r0 = std::sqrt(b), r1 = std::sqrt(2.0 * b);
            div_bad += !same(divide(x, b), q);
            root_bad += !same(root(b), r0) + !same(root(2.0 * b), r1);
        }
        std::printf("seeds %+d ulp: %ld quotients and %ld roots differ\n", u, div_bad, root_bad);
        total += div_bad + root_bad;
    }
    return total != 0;
}
