// phase_barrier_check.cpp -- the barriers between the phases of a
// characteristic field (csrc/physics_exact.cuh char_pair, lattice_fp64.cuh
// char_node) counted on the host, one thread of a block after the other: a
// block-wide barrier is only defined if every thread meets it, so threads
// past the range and threads whose node has no face must count as many as
// the others.  Lattices with non-periodic directions (nodes without a face),
// a range that ends inside a block, and field by field; a face's results are
// those of a call without barriers.  Prints the threads that counted
// differently; exit code 1 if there is any.
#include <math.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

// the device's built-ins that the headers name (no code of them runs here
// but the bit casts)
static struct { unsigned x = 0; } threadIdx;
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dsub_rn(double a, double b) { return a - b; }
static inline float __double2float_rn(double x) { return (float)x; }
static inline float __int2float_rn(int x) { return (float)x; }
static inline uint32_t __float_as_uint(float f)
{
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}
static inline float __uint_as_float(uint32_t u)
{
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
static inline int __clzll(long long x) { return x ? __builtin_clzll((unsigned long long)x) : 64; }
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }
static inline float __ldg(const float *p) { return *p; }
static inline double __ldg(const double *p) { return *p; }
static inline double __longlong_as_double(long long u)
{
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}
static inline long long __double_as_longlong(double x)
{
    long long u;
    std::memcpy(&u, &x, 8);
    return u;
}
template <class T>
static inline T __shfl_xor_sync(unsigned, T x, int) { return x; }
static inline void __syncthreads() {}
static inline void atomicOr(unsigned *p, unsigned v) { *p |= v; }

#define __noinline__ __attribute__((noinline))
#include "lattice_fp64.cuh"

using namespace cfd;

struct CountSync {
    int *n;
    void operator()() const { ++*n; }
};

// One field of every face of a lattice in blocks of `threads` over nodes
// 0 .. n1 - 1; per: periodic directions.
static long check(int ni, int nj, int nk, int per, int n1, int threads)
{
    const int N = ni * nj * nk;
    std::vector<double> Q(5 * N), kn(9 * N), fs((size_t)3 * kFaceScratch * N, 1.0), want = fs;
    uint64_t s = 12345;
    auto rnd = [&]() { return (double)((s = s * 6364136223846793005ull + 1442695040888963407ull) >> 40) / (1 << 24) + 0.5; };
    for (double &x : Q) x = rnd();
    for (double &x : kn) x = rnd();
    LatView g{};
    g.ni = ni;
    g.nj = nj;
    g.nk = nk;
    g.N = N;
    g.per = per;
    g.P.eps = 1e-7;
    g.Q = Q.data();
    g.kn = kn.data();
    for (size_t i = 0; i < fs.size(); ++i) want[i] = fs[i] = rnd();
    const FaceScratch A{fs.data(), 0, N}, B{want.data(), 0, N};
    long bad = 0;
    for (int d = 0; d < 3; ++d)
        for (int q = 0; q < 5; ++q) {
            for (int b0 = 0; b0 < n1; b0 += threads) {
                int most = 0;
                std::vector<int> count(threads, 0);
                for (int t = 0; t < threads; ++t) {
                    ex::char_node(g, A, b0 + t, d, q, b0 + t < n1, CountSync{&count[t]});
                    if (count[t] > most) most = count[t];
                }
                for (int c : count) bad += most == 0 || c != most;
            }
            for (int n = 0; n < n1; ++n) ex::char_node(g, B, n, d, q, true);
        }
    for (size_t i = 0; i < fs.size(); ++i) bad += std::memcmp(&fs[i], &want[i], 8) != 0;
    std::printf("%d x %d x %d, periodic %d, %d nodes in blocks of %d: %ld threads out of step\n", ni, nj, nk, per, n1,
                threads, bad);
    return bad;
}

int main()
{
    long bad = 0;
    for (int threads : {32, 256}) {
        bad += check(7, 6, 5, 7, 7 * 6 * 5, threads);    // every node has its faces; the last block is ragged
        bad += check(12, 9, 7, 1, 12 * 9 * 7, threads);  // walls along j and k
        bad += check(8, 8, 8, 0, 300, threads);          // walls everywhere, a range that ends in a block
    }
    return bad != 0;
}
