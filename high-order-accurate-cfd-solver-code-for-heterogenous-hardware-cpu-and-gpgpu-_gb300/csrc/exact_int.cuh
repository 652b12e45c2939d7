// exact_int.cuh -- binary64 products and quotients on the integer pipe, in
// groups: the IEEE results (round to nearest even) of several independent
// operations computed without a branch between them.
//
// GB300 issues an FP64 instruction of a warp every 64 clocks per scheduler
// and an integer one every two, so a rounded product of about twenty-five
// integer instructions runs beside the FP64 pipe at its own price, and a
// quotient at half the price of a division on it -- provided the warps in
// flight hide the latency of the integer chains.  A test and a branch after
// each operation would order the chains one after the other; here a group's
// operations share one test, and the instructions of all of them overlap.
//
// Plain case: operands in [2^-255, 2^257), so that no result leaves the
// normal range, and (products) no exact tie.  Everything else is resolved
// operand by operand in an out-of-line branch: exact zeros, which flows
// that stay two-dimensional carry at every node, then the FP64 instruction.
// Host code gets the same routines for the checks.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define CFD_XI_HD __host__ __device__ __forceinline__
#else
#define CFD_XI_HD inline
#endif

namespace cfd {
namespace xi {

CFD_XI_HD uint32_t hi32(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return (uint32_t)(u >> 32);
#endif
}

CFD_XI_HD uint32_t lo32(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return (uint32_t)u;
#endif
}

CFD_XI_HD double words(uint32_t hi, uint32_t lo)
{
#if defined(__CUDA_ARCH__)
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo;
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}

CFD_XI_HD uint32_t umulhi(uint32_t a, uint32_t b)
{
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// high word of (hi:lo) << s, 0 <= s < 32
CFD_XI_HD uint32_t funnel_l(uint32_t lo, uint32_t hi, uint32_t s)
{
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}

// The host's seeds of the reciprocal and the reciprocal root; a check may put
// worse ones in their place, as far off as the device's may be.
#ifndef CFD_XI_HOST_RCP
#define CFD_XI_HOST_RCP(m) (1.0f / (m))
#endif
#ifndef CFD_XI_HOST_RSQRT
#define CFD_XI_HOST_RSQRT(m) ((float)(1.0 / std::sqrt((double)(m))))
#endif

constexpr uint32_t kMark = 0x60000000u;

// Nonzero for the high word of an operand outside [2^-255, 2^257) (biased
// exponent outside [768, 1279]: plus 256, its two leading bits are not 10);
// zeros, subnormals, infinities and NaN among them.
CFD_XI_HD uint32_t mark_of(uint32_t hi) { return ((hi + 0x10000000u) ^ 0x40000000u) & kMark; }

// An operand unpacked: the 53-bit significand left-aligned in 64 bits is h
// (its top 32 bits, leading bit set) and the 21 bits below, l; e holds the
// sign and the biased exponent where the double's high word does.  The bits
// kMark of l mark an operand outside the plain case.  An operand of
// several operations is unpacked once.
struct Fac {
    uint32_t h, l, e;
};

CFD_XI_HD Fac fac(double x)
{
    const uint32_t hi = hi32(x), lo = lo32(x);
    return {(hi << 11) | (lo >> 21) | 0x80000000u, (lo & 0x1fffffu) | mark_of(hi), hi & 0xfff00000u};
}

// A marked operand that is a zero; an operand that is not Inf or NaN.
CFD_XI_HD bool is_zero(Fac f) { return ((f.h << 1) | (f.l & 0x1fffffu) | (f.e << 1)) == 0u; }
CFD_XI_HD bool is_finite(Fac f) { return (f.e & 0x7ff00000u) != 0x7ff00000u; }

CFD_XI_HD double unpacked(Fac f) { return words(f.e | ((f.h >> 11) & 0xfffffu), (f.h << 21) | (f.l & 0x1fffffu)); }

// ---------------------------------------------------------- products ---
// The significands' product is
//   P = ha hb 2^42 + (ha lb + la hb) 2^21 + la lb.
// mid = ha lb + la hb + floor(la lb / 2^21) and T = ha hb + floor(mid /
// 2^21) give P exactly down to 2^21: T = floor(P / 2^42), and the low 21
// bits of mid are the next ones.  T's leading bit is bit 63 or 62, so the
// result is T without its low n = 11 or 10 bits, rounded up when the
// dropped part is above half.  rem holds those n bits at the top of a word
// and the bits of mid below them; what it leaves out is positive and less
// than its last bit (n = 11) or its last two (n = 10, where the last is 0),
// so rem decides except at exactly half, where the product may be a tie:
// bad is set there and for marked operands.
CFD_XI_HD uint32_t mul_words(Fac a, Fac b, uint32_t &hi, uint32_t &lo)
{
    const uint64_t mid = (uint64_t)a.h * b.l + ((uint64_t)a.l * b.h + umulhi(a.l << 11, b.l));
    const uint64_t T = (uint64_t)a.h * b.h + (mid >> 21);
    const uint32_t n = 10u + (uint32_t)(T >> 63);
    const uint32_t rem = funnel_l((uint32_t)mid << 11, (uint32_t)T, 32u - n);
    const uint64_t M = (T >> n) + (rem >> 31);
    hi = (uint32_t)(M >> 32) + a.e + b.e + (n << 20) - (1034u << 20);   // exponents add; M's hidden bit adds one
    lo = (uint32_t)M;
    return ((a.l | b.l) & kMark) | (uint32_t)(rem == 0x80000000u);
}

// One product outside the plain case, out of line on the unpacked words
// (unpacking or testing them at each call costs the flows that never come
// here: TGV 128^3 1.5 ms a step): zeros of the right sign for a zero times a
// finite operand, which flows that stay two-dimensional carry at every node,
// else the FP64 multiply.
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
    double
    mul_rare(Fac a, Fac b)
{
    if ((is_zero(a) || is_zero(b)) && is_finite(a) && is_finite(b)) return words((a.e ^ b.e) & 0x80000000u, 0u);
#if defined(__CUDA_ARCH__)
    return __dmul_rn(unpacked(a), unpacked(b));
#else
    volatile double r = unpacked(a) * unpacked(b);
    return r;
#endif
}

// r[i] = a[i] * b[i]
template <int N>
CFD_XI_HD void mul_n(const Fac (&a)[N], const Fac (&b)[N], double (&r)[N])
{
    uint32_t hi[N], lo[N], bad[N], any = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        bad[i] = mul_words(a[i], b[i], hi[i], lo[i]);
        any |= bad[i];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = words(hi[i], lo[i]);
    if (__builtin_expect(any != 0u, 0)) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (bad[i]) r[i] = mul_rare(a[i], b[i]);
    }
}

CFD_XI_HD double mul(double a, double b)
{
    const Fac fa[1] = {fac(a)}, fb[1] = {fac(b)};
    double r[1];
    mul_n(fa, fb, r);
    return r[0];
}

// x[i] = x[i]^2
template <int N>
CFD_XI_HD void sq_n(double (&x)[N])
{
    Fac f[N];
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = fac(x[i]);
    mul_n(f, f, x);
}

// x * C 2^K for an odd constant 3 <= C <= 63 and |K| <= 8: the significand
// times C is exact in 59 bits and is rounded in place (half less one plus
// the result's last bit added before the shift), so ties need no branch.
// The returned mark is set outside the plain case.
template <int C, int K>
CFD_XI_HD uint32_t small_words(double x, uint32_t &hi, uint32_t &lo)
{
    static_assert(C >= 3 && C <= 63 && (C & 1) && K >= -8 && K <= 8, "small_words");
    constexpr uint32_t lc = C >= 32 ? 5u : C >= 16 ? 4u : C >= 8 ? 3u : C >= 4 ? 2u : 1u;   // floor(log2 C)
    const uint32_t xh = hi32(x), xl = lo32(x);
    const uint64_t X = ((uint64_t)((xh & 0xfffffu) | 0x100000u) << 32) | xl;
    const uint64_t T = X * (uint32_t)C;
    const uint32_t sh = lc + (uint32_t)(T >> (53u + lc));
    const uint64_t M = (T + (((1u << sh) >> 1) - 1u) + (((uint32_t)T >> sh) & 1u)) >> sh;
    hi = (uint32_t)(M >> 32) + (xh & 0xfff00000u) + (sh << 20) + (uint32_t)((K - 1) * (1 << 20));
    lo = (uint32_t)M;
    return mark_of(xh);
}

// small_words' result, or x c (c = C 2^K) where it is marked.
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
    double
    small_rare(double x, double c)
{
    if (((hi32(x) << 1) | lo32(x)) == 0u) return x;
#if defined(__CUDA_ARCH__)
    return __dmul_rn(x, c);
#else
    volatile double r = x * c;
    return r;
#endif
}

CFD_XI_HD double small_or(uint32_t mark, uint32_t hi, uint32_t lo, double x, double c)
{
    return __builtin_expect(mark != 0u, 0) ? small_rare(x, c) : words(hi, lo);
}

// --------------------------------------------------------- quotients ---
// A divisor b = +-B 2^(e - 1075) (B its 53-bit significand, beta = B / 2^52
// in [1, 2)) with Y, an approximation of 2^64 / beta that Y <= 2^64 / beta
// < Y + 4 (for beta = 1: Y = 2^64 - 1).  A float reciprocal of B's top 24
// bits, clamped to [1/2, 1 - 2^-24], seeds it: r = S 2^-24 with eps = 1 -
// beta r = E / 2^76 exactly, E = 2^76 - S B, and |eps| < 2^-21.4 (the seed
// within 2^-23, which for a divisor just below 2 may be under 1/2; the dropped
// bits of B within 2^-23), so |E| < 2^54.6 and its low
// 64 bits are E.  Then 2^64 / beta = S 2^40 (1 + eps + eps^2 + ...) and
//   Y = S 2^40 + floor(S (E + floor(E^2 / 2^76)) / 2^36) - 2:
// the terms left out are below 2^-64.2 / (1 - eps) relative, under one unit
// of Y either way, E^2 from E's top bits is within 2^-8 of a unit, and the
// floors lose less than one more.
struct Divisor {
    uint32_t yh, yl;   // Y
    uint32_t bh, bl;   // the double's words; bit-for-bit the divisor
};

CFD_XI_HD float seed_rcp(float m)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(m));   // within 2^-23 for m in [1, 2)
    return r;
#else
    return CFD_XI_HOST_RCP(m);
#endif
}

CFD_XI_HD Divisor divisor(double b)
{
    const uint32_t bh = hi32(b), bl = lo32(b);
    const uint32_t mb = ((bh << 3) & 0x7fffffu) | (bl >> 29) | 0x3f800000u;
#if defined(__CUDA_ARCH__)
    const uint32_t rb = __float_as_uint(fmaxf(fminf(seed_rcp(__uint_as_float(mb)), 0.99999994f), 0.5f));
#else
    float m, r;
    std::memcpy(&m, &mb, 4);
    r = seed_rcp(m);
    r = r < 0.99999994f ? r : 0.99999994f;
    r = r > 0.5f ? r : 0.5f;
    uint32_t rb;
    std::memcpy(&rb, &r, 4);
#endif
    const uint32_t S = (rb & 0x7fffffu) | 0x800000u;
    const uint64_t B = ((uint64_t)((bh & 0xfffffu) | 0x100000u) << 32) | bl;
    const int64_t E = (int64_t)(0ULL - B * S);
    const int32_t Eh = (int32_t)(E >> 24);
    const int64_t G = E + (((int64_t)Eh * Eh) >> 28);
    const int64_t W = (int64_t)(int32_t)(G >> 32) * (int32_t)S + (int64_t)umulhi(S, (uint32_t)G) - 32;
    const uint64_t Y = ((uint64_t)(S << 8) << 32) + (uint64_t)(W >> 4);
    return {(uint32_t)(Y >> 32), (uint32_t)Y, bh, bl};
}

// x / b.  With X = x.h 2^21 + x.l, T = x.h yh + floor(x.h yl / 2^32) +
// floor(2^11 x.l yh / 2^32) is at most X Y / 2^53 and less than three below
// it, and Y's own error moves X Y / 2^53 by less than four: the exact
// quotient of the significands, V = X 2^64 / (beta 2^53), lies in [T, T +
// 7).  T's leading bit is bit 63 or 62; without its low n = 11 or 10 bits it
// is M, the quotient's 53 bits or (near the end of a step) one less.  Round
// to nearest takes M or M + 1 as V 2^-n lies below or above M + 1/2 --
// never on it, since a quotient is no midpoint -- and that is the sign of
//   D = X 2^(64 - n) - (2 M + 1) B
// (|D| < 2^55, so the low 64 bits give it; X 2^(64 - n) has only its high
// word).  When T falls just short of 2^63 and V does not (X >= B), the
// step M + 1 carries into the exponent, as it should.
CFD_XI_HD uint32_t quot_words(Fac x, const Divisor &d, uint32_t &hi, uint32_t &lo)
{
    const uint64_t T = (uint64_t)x.h * d.yh + ((uint64_t)umulhi(x.h, d.yl) + umulhi(x.l << 11, d.yh));
    const uint32_t n = 10u + (uint32_t)(T >> 63);
    const uint64_t C = (T >> (n - 1u)) | 1u;   // 2 M + 1
    const uint32_t Bh = (d.bh & 0xfffffu) | 0x100000u;
    const uint64_t p = (uint64_t)(uint32_t)C * d.bl;
    const uint32_t ph = (uint32_t)(p >> 32) + (uint32_t)C * Bh + (uint32_t)(C >> 32) * d.bl;
    const uint32_t xl = (x.h << 21) | x.l;     // X's low word
    const uint64_t D = ((uint64_t)(xl << (32u - n)) << 32) - (((uint64_t)ph << 32) | (uint32_t)p);
    const uint64_t M = (C >> 1) + (uint32_t)(~(uint32_t)(D >> 32) >> 31);
    hi = (uint32_t)(M >> 32) + x.e - (d.bh & 0xfff00000u) + (n << 20) + (1011u << 20);
    lo = (uint32_t)M;
    return (x.l | mark_of(d.bh)) & kMark;
}

// One quotient outside the plain case: IEEE 754's exact results for zero
// and infinite operands (signs exclusive-ored), else the division.
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
    double
    quot_rare(double x, double b)
{
    const uint32_t xh = hi32(x), bh = hi32(b), ax = xh & 0x7fffffffu, ab = bh & 0x7fffffffu;
    const uint32_t s = (xh ^ bh) & 0x80000000u;
    const bool x0 = (ax | lo32(x)) == 0u, b0 = (ab | lo32(b)) == 0u;
    const bool xf = ax < 0x7ff00000u, bf = ab < 0x7ff00000u;             // finite
    const bool xinf = ax == 0x7ff00000u && lo32(x) == 0u, binf = ab == 0x7ff00000u && lo32(b) == 0u;
    if ((x0 && bf && !b0) || (xf && binf)) return words(s, 0u);
    if ((b0 && xf && !x0) || (xinf && bf)) return words(s | 0x7ff00000u, 0u);
#if defined(__CUDA_ARCH__)
    return __ddiv_rn(x, b);
#else
    volatile double r = x / b;
    return r;
#endif
}

// x[i] = x[i] / b
template <int N>
CFD_XI_HD void quot_n(double (&x)[N], const Divisor &d)
{
    uint32_t hi[N], lo[N], bad[N], any = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        bad[i] = quot_words(fac(x[i]), d, hi[i], lo[i]);
        any |= bad[i];
    }
    if (__builtin_expect(any != 0u, 0)) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (bad[i]) {
                const double r = quot_rare(x[i], words(d.bh, d.bl));
                hi[i] = hi32(r);
                lo[i] = lo32(r);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = words(hi[i], lo[i]);
}

// x[i] / b[i]
template <int N>
CFD_XI_HD void div_n(double (&x)[N], const double (&b)[N])
{
    uint32_t hi[N], lo[N], bad[N], any = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        bad[i] = quot_words(fac(x[i]), divisor(b[i]), hi[i], lo[i]);
        any |= bad[i];
    }
    if (__builtin_expect(any != 0u, 0)) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (bad[i]) {
                const double r = quot_rare(x[i], b[i]);
                hi[i] = hi32(r);
                lo[i] = lo32(r);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = words(hi[i], lo[i]);
}

CFD_XI_HD double divide(double x, double b)
{
    double q[1] = {x};
    const double d[1] = {b};
    div_n(q, d);
    return q[0];
}

// ------------------------------------------------------ square roots ---
// x = m 2^(2 k), m = A / 2^52 in [1, 4) (A the significand, doubled when the
// exponent is odd).  A float reciprocal root of m's top bits, clamped to
// [1/2, 1 - 2^-24], is r = R 2^-24 with eps = 1 - m r^2, |eps| < 2^-20.7 (two
// ulps of r and the bits dropped from m).  Then
//   sqrt(m) = m r (1 - eps)^(-1/2) = m r (1 + eps / 2 + 3 eps^2 / 8 + ...)
// to 2^-64 relative; G = m r^2 2^62, c = (eps / 2 + 3 eps^2 / 8) 2^63 and
// T = m r (1 + c) 2^62 are evaluated with the low products left out, which
// moves T by less than 32 either way, so with 64 taken off T lies below
// sqrt(m) 2^62 by less than 96.  M = floor(T / 2^10) is then the root's 53
// bits or one less; round to nearest takes M + 1 where sqrt(m) 2^52 > M +
// 1/2 (a root is no midpoint), that is where
//   D = A 2^54 - (2 M + 1)^2 > 0   (|D| < 2^56: the low 64 bits give it).
CFD_XI_HD float seed_rsqrt(float m)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(m));
    return r;
#else
    return CFD_XI_HOST_RSQRT(m);
#endif
}

CFD_XI_HD uint32_t sqrt_words(double x, uint32_t &hi, uint32_t &lo)
{
    const uint32_t xh = hi32(x), xl = lo32(x);
    const uint32_t odd = ~(xh >> 20) & 1u;   // the unbiased exponent is odd
    const uint64_t A = (((uint64_t)((xh & 0xfffffu) | 0x100000u) << 32) | xl) << odd;
    const uint32_t mb = (((xh << 3) & 0x7fffffu) | (xl >> 29)) + 0x3f800000u + (odd << 23);
#if defined(__CUDA_ARCH__)
    const uint32_t rb = __float_as_uint(fmaxf(fminf(seed_rsqrt(__uint_as_float(mb)), 0.99999994f), 0.5f));
#else
    float m, r;
    std::memcpy(&m, &mb, 4);
    r = seed_rsqrt(m);
    r = r < 0.99999994f ? r : 0.99999994f;
    r = r > 0.5f ? r : 0.5f;
    uint32_t rb;
    std::memcpy(&rb, &r, 4);
#endif
    const uint32_t R = (rb & 0x7fffffu) | 0x800000u;
    const uint64_t P = ((uint64_t)R * R) << 16;                  // r^2 2^64
    const uint64_t A10 = A << 10;                                // m 2^62
    const uint32_t ph = (uint32_t)(P >> 32), pl = (uint32_t)P, ah = (uint32_t)(A10 >> 32), al = (uint32_t)A10;
    const uint64_t G = (uint64_t)ph * ah + ((uint64_t)umulhi(ph, al) + umulhi(pl, ah));
    const int64_t E = (int64_t)((1ULL << 62) - G);               // eps 2^62
    const int32_t eh = (int32_t)(E >> 12);
    const int64_t c = E + ((3 * ((int64_t)eh * eh)) >> 40);      // |c| < 2^41.5
    const uint64_t W = ((uint64_t)(uint32_t)(A >> 32) * R << 18) + ((uint64_t)(uint32_t)A * R >> 14);   // m r 2^62
    const int32_t ch = (int32_t)(c >> 32);
    const uint32_t wh = (uint32_t)(W >> 32), wl = (uint32_t)W;
    const int64_t V = (int64_t)ch * (int64_t)wh + (int64_t)umulhi(wh, (uint32_t)c) + (((int64_t)ch * (int64_t)wl) >> 32);
    const uint64_t T = W + (uint64_t)(V * 2) - 64u;
    const uint64_t C = (T >> 9) | 1u;                            // 2 M + 1
    const uint32_t cl = (uint32_t)C, chi = (uint32_t)(C >> 32);
    const uint64_t q = (uint64_t)cl * cl;
    const uint64_t sq = q + ((uint64_t)(2u * cl * chi) << 32);
    const uint64_t D = ((uint64_t)((uint32_t)A << 22) << 32) - sq;
    const uint64_t M = (C >> 1) + (uint32_t)(~(uint32_t)(D >> 32) >> 31);
    hi = (uint32_t)(M >> 32) + ((((xh >> 20) + 1u) >> 1) << 20) + (510u << 20);
    lo = (uint32_t)M;
    return mark_of(xh) | (xh & 0x80000000u);
}

// One root outside the plain case: zeros are their own, else the instruction.
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
    double
    sqrt_rare(double x)
{
    if (((hi32(x) << 1) | lo32(x)) == 0u) return x;
#if defined(__CUDA_ARCH__)
    return __dsqrt_rn(x);
#else
    return std::sqrt(x);
#endif
}

// x[i] = sqrt(x[i])
template <int N>
CFD_XI_HD void sqrt_n(double (&x)[N])
{
    uint32_t hi[N], lo[N], bad[N], any = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        bad[i] = sqrt_words(x[i], hi[i], lo[i]);
        any |= bad[i];
    }
    if (__builtin_expect(any != 0u, 0)) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (bad[i]) {
                const double r = sqrt_rare(x[i]);
                hi[i] = hi32(r);
                lo[i] = lo32(r);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = words(hi[i], lo[i]);
}

CFD_XI_HD double root(double x)
{
    double r[1] = {x};
    sqrt_n(r);
    return r[0];
}

}  // namespace xi
}  // namespace cfd
