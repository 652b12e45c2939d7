// lattice_mixed.cuh -- per-node operations of the mixed-precision lattice
// stage, written for a part whose FP64 rate is a small fraction of its FP32
// rate.
//
// State: each conserved value of U0/U1/U2 is carried as hi + lo, two FP32
// numbers (about 48 significant bits; double-float arithmetic after Dekker,
// "A floating-point technique for extending the available precision", 1971,
// with the FMA-based exact product).  The RK3 accumulation runs in that
// arithmetic on the FP32 pipe.
// FP32: characteristic projection, WENO5, LLF, face and node fluxes, the
// viscous/SGS fluxes, the right-hand side sum, and the primitives derived
// from the state each stage (rounded once from hi/lo quotients).  On a
// lattice with ghost layers the same loc-code branches as the FP64 form,
// and the boundary routine on the hi/lo state (bc_target).
// FP64 only at the boundary: FLOW in (kPrepFromFlow) and FLOW/U out.
// Include only from translation units compiled with FMA contraction and
// approximate FP32 division/square root; the hi/lo routines below use
// explicit fmaf and plain additions, which contraction leaves exact.
#pragma once

#include "boundary.h"
#include "face_tile.cuh"
#include "lattice.cuh"
#include "physics_x2.cuh"

namespace cfd {
namespace mx {

struct dfl {
    float h, l;
};

// s + e == a + b exactly (Knuth's two-sum)
__device__ __forceinline__ dfl two_sum(float a, float b)
{
    const float s = a + b;
    const float bb = s - a;
    const float e = (a - (s - bb)) + (b - bb);
    return {s, e};
}

// s + e == a + b exactly when |a| >= |b| or a == 0 (Dekker's fast two-sum)
__device__ __forceinline__ dfl quick_two_sum(float a, float b)
{
    const float s = a + b;
    return {s, b - (s - a)};
}

__device__ __forceinline__ dfl df_add(dfl x, dfl y)
{
    const dfl s = two_sum(x.h, y.h);
    const dfl t = two_sum(x.l, y.l);
    dfl v = quick_two_sum(s.h, s.l + t.h);
    return quick_two_sum(v.h, t.l + v.l);
}

// x * c, c given as hi + lo
__device__ __forceinline__ dfl df_mul(dfl x, dfl c)
{
    const float p = x.h * c.h;
    float e = fmaf(x.h, c.h, -p);
    e = fmaf(x.h, c.l, fmaf(x.l, c.h, e));
    return quick_two_sum(p, e);
}

// x * c rounded once to FP32
__device__ __forceinline__ float df_mul_f(dfl x, dfl c)
{
    return fmaf(x.h, c.h, fmaf(x.h, c.l, __fmul_rn(x.l, c.h)));
}

// a / b rounded to FP32 (within about one ulp), r an approximation of 1/b.h
__device__ __forceinline__ float df_div_f(dfl a, dfl b, float r)
{
    const float q = a.h * r;
    const float rem = fmaf(-q, b.h, a.h) + fmaf(-q, b.l, a.l);
    return fmaf(rem, r, q);
}

// a / b as hi + lo (error near 2^-44 relative)
__device__ __forceinline__ dfl df_div(dfl a, dfl b, float r)
{
    const float q = df_div_f(a, b, r);
    const float p = q * b.h;
    const float pe = fmaf(q, b.h, -p);
    // remainder a - q*b, then one correction step
    const float rem = ((a.h - p) - pe) + fmaf(-q, b.l, a.l);
    return quick_two_sum(q, __fmul_rn(rem, r));
}

// 1/3 as hi + lo
constexpr float kThirdH = (float)(1.0 / 3.0);
constexpr float kThirdL = (float)(1.0 / 3.0 - (double)(float)(1.0 / 3.0));
// gamma - 1 = 0.4 as hi + lo
constexpr float kGm1H = (float)0.4;
constexpr float kGm1L = (float)(0.4 - (double)(float)0.4);

__device__ __forceinline__ void load_state(const LatView &g, int q, int n, dfl Un[5])
{
    const int N = g.N;
    const float *W = lat_W(g, q);
#pragma unroll
    for (int c = 0; c < 5; ++c) Un[c] = {lat_at(W, c, N, n), lat_at(W, 5 + c, N, n)};
}

__device__ __forceinline__ void store_state(const LatView &g, int q, int n, const dfl Un[5])
{
    const int N = g.N;
    float *W = lat_W(g, q);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        lat_at(W, c, N, n) = Un[c].h;
        lat_at(W, 5 + c, N, n) = Un[c].l;
    }
}

// U_Q of the next stage from the state Un (= det * Q): the inputs of the
// face stage -- Q, the Roe inputs (u, v, w, sqrt(rho), H) and the pressure
// (prim32); the viscous pass takes rho from Q and u, v, w from the Roe
// inputs, and FLOW leaves through flow_out_node.
__device__ __forceinline__ void derive(const LatView &g, int n, const dfl Un[5])
{
    const int N = g.N;
    const dfl idet = {lat_at(g.idet32, 0, N, n), lat_at(g.idet32, 1, N, n)};
    const float r0 = frcp(Un[0].h);
    const float rho = df_mul_f(Un[0], idet);
    const float u = df_div_f(Un[1], Un[0], r0), v = df_div_f(Un[2], Un[0], r0), w = df_div_f(Un[3], Un[0], r0);
    const float ke = __fmul_rn(0.5f, dot3(u, u, v, v, w, w));
    const dfl q4 = df_div(Un[4], Un[0], r0);   // E / rho
    const dfl e2 = df_add(q4, {-ke, 0.0f});      // internal energy e
    const dfl rho2 = df_mul(Un[0], idet);
    const float p = df_mul_f(df_mul(rho2, e2), {kGm1H, kGm1L});
    const float irho = frcp(rho);
    const float pr = __fmul_rn(p, irho);
    lat_at(g.prim32, LF_P, N, n) = p;
    if (!(isfinite(rho) && isfinite(u) && isfinite(v) && isfinite(w) && isfinite(p))) atomicOr(g.flags, 2u);
    const float E = df_mul_f(Un[4], idet);
    lat_at(g.Q32, 0, N, n) = rho;
    lat_at(g.Q32, 1, N, n) = df_mul_f(Un[1], idet);
    lat_at(g.Q32, 2, N, n) = df_mul_f(Un[2], idet);
    lat_at(g.Q32, 3, N, n) = df_mul_f(Un[3], idet);
    lat_at(g.Q32, 4, N, n) = E;
    lat_at(g.R32, 0, N, n) = u;
    lat_at(g.R32, 1, N, n) = v;
    lat_at(g.R32, 2, N, n) = w;
    lat_at(g.R32, 3, N, n) = fsqrt(rho);
    lat_at(g.R32, 4, N, n) = q4.h + (q4.l + pr);     // H = E/rho + p/rho
}

// U_Q from the FP64 FLOW (after an upload): U = det * Q(FLOW) in FP64, split
// into hi + lo in slot q, then derive.
__device__ __forceinline__ void init_node(const LatView &g, int n, int q)
{
    const int N = g.N;
    const double rho = g.prim9[LF_RHO * N + n], u = g.prim9[LF_U * N + n], v = g.prim9[LF_V * N + n],
                 w = g.prim9[LF_W * N + n], p = g.prim9[LF_P * N + n];
    const double D = g.det[n];
    const double E = xi::divide(p, 0.4) + 0.5 * rho * (u * u + v * v + w * w);
    const double U[5] = {D * rho, D * rho * u, D * rho * v, D * rho * w, D * E};
    dfl Un[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) emu::hi_lo(U[c], Un[c].h, Un[c].l);
    store_state(g, q, n, Un);
    g.prim32[LF_MU * N + n] = emu::d2f(g.prim9[LF_MU * N + n]);
    derive(g, n, Un);
}

// U_Q from the state in slot src, copied to slot dst (a stage run out of the
// usual order: U_dst = det * Q(FLOW) with FLOW the current state).
__device__ __forceinline__ void prep_node(const LatView &g, int n, int src, int dst)
{
    dfl Un[5];
    load_state(g, src, n, Un);
    if (src != dst) store_state(g, dst, n, Un);
    derive(g, n, Un);
}

// Derivative of branch b (physics.cuh visc_branch) from the six neighbour
// differences dl[m] = f[m+1] - f[m] of the values at offsets -3..3: every
// formula rewritten as a sum of neighbour differences, which the hi/lo
// state gives to FP32 accuracy.
__device__ __forceinline__ float branch_deriv_diff(int b, const float dl[6])
{
    switch (b) {
    case 1: return (1.0f / 6.0f) * (11.0f * dl[2] - 7.0f * dl[1] + 2.0f * dl[0]);
    case 2: return (1.0f / 6.0f) * (11.0f * dl[3] - 7.0f * dl[4] + 2.0f * dl[5]);
    case 3: return (1.0f / 6.0f) * (2.0f * dl[3] + 5.0f * dl[2] - dl[1]);
    case 4: return (1.0f / 6.0f) * (2.0f * dl[2] + 5.0f * dl[3] - dl[4]);
    case 5: return (1.0f / 12.0f) * (8.0f * (dl[2] + dl[3]) - (dl[1] + dl[2] + dl[3] + dl[4]));
    default: return 0.0f;
    }
}

// Viscous + MTS SGS fluxes from slot q.  Derivatives of U from hi/lo
// differences (exact hi differences for neighbours within a factor of two):
// central on a periodic lattice (LOC = false), the reference's loc-code
// branches on a lattice with loc codes (LOC = true; zero at ghosts);
// everything else in FP32.
template <bool LOC>
__device__ __forceinline__ void visc_node(const LatView &g, int n, int q)
{
    const int N = g.N;
    const float *W = lat_W(g, q);
    int i, j, k;
    lat_ijk(g, n, i, j, k);
    float dU[3][5], KS[3], Ui[5];
    auto filtered = [](float a, float b, float c) { return fmaf(0.25f, a + c, __fmul_rn(0.5f, b)); };
    const bool ghost = LOC && lat_ghost(g, n);
    const unsigned lflag = (LOC && g.locflag) ? g.locflag[n] : 7u;
#pragma unroll
    for (int c = 0; c < 5; ++c) Ui[c] = W[c * N + n];
    const float r0 = frcp(Ui[0]);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int m2 = lat_step(g, i, j, k, d, -2), m1 = lat_step(g, i, j, k, d, -1), p1 = lat_step(g, i, j, k, d, 1),
                  p2 = lat_step(g, i, j, k, d, 2);
        if (ghost) {
#pragma unroll
            for (int c = 0; c < 5; ++c) dU[d][c] = 0.0f;
        } else if (!LOC || !lat_locdir(g, d) || !((lflag >> d) & 1u)) {
            const unsigned o2 = 4u * m2, o1 = 4u * m1, q1 = 4u * p1, q2 = 4u * p2;
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                // the state slot is read-only in this pass: non-coherent loads
                const float *H = W + (size_t)c * N, *L = W + (size_t)(5 + c) * N;
                const float d1 = (lat_ldg(H, q1) - lat_ldg(H, o1)) + (lat_ldg(L, q1) - lat_ldg(L, o1));
                const float d2 = (lat_ldg(H, q2) - lat_ldg(H, o2)) + (lat_ldg(L, q2) - lat_ldg(L, o2));
                dU[d][c] = __fmul_rn(1.0f / 12.0f, fmaf(8.0f, d1, -d2));
            }
        } else {
            int s[7], L7[7];
#pragma unroll
            for (int o = 0; o < 7; ++o) {
                s[o] = lat_step(g, i, j, k, d, o - 3);
                L7[o] = g.loc8[s[o]];
            }
            const int b = visc_branch(L7);
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const float *H = W + c * N, *L = W + (5 + c) * N;
                float dl[6];
#pragma unroll
                for (int m = 0; m < 6; ++m) dl[m] = (H[s[m + 1]] - H[s[m]]) + (L[s[m + 1]] - L[s[m]]);
                dU[d][c] = branch_deriv_diff(b, dl);
            }
        }
        const float *Wd = W + (size_t)(d + 1) * N;
        const int c = d + 1;
        const float um = lat_ldg(Wd, 4u * m1), up = lat_ldg(Wd, 4u * p1);
        const float rm = lat_ldg(W, 4u * m1), rp = lat_ldg(W, 4u * p1);
        const float dlt = fmaf(Ui[c], r0, -qdiv(filtered(um, Ui[c], up), filtered(rm, Ui[0], rp)));
        KS[d] = fabsf(dlt);
    }
    float m[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) m[c] = lat_at(g.node32, c, N, n);
    const float prim[5] = {lat_at(g.Q32, 0, N, n), lat_at(g.R32, 0, N, n), lat_at(g.R32, 1, N, n), lat_at(g.R32, 2, N, n),
                           lat_at(g.prim32, LF_P, N, n)};
    float Fv[5], Ev[5], Gv[5], mu;
    viscous_node_flux(dU, Ui, m, lat_at(g.node32, 9, N, n), lat_at(g.node32, 10, N, n), prim, KS, g.P, Fv, Ev, Gv, mu);
#pragma unroll
    for (int c = 1; c < 5; ++c) {   // mass has no viscous flux: component 0 stays as it was zeroed
        lat_at(g.V32, c, N, n) = Fv[c];
        lat_at(g.V32, 5 + c, N, n) = Ev[c];
        lat_at(g.V32, 10 + c, N, n) = Gv[c];
    }
    lat_at(g.prim32, LF_MU, N, n) = mu;
}

__device__ __forceinline__ void mu_node(const LatView &g, int n, int q)
{
    const int N = g.N;
    const float *W = lat_W(g, q);
    const float U0 = W[n], iU0 = qdiv(1.0f, U0);
    const float uu = W[N + n] * iU0, vv = W[2 * N + n] * iU0, ww = W[3 * N + n] * iU0;
    const float mach = (float)g.P.mach;
    const float d_temp = 1.4f * mach * mach * 0.4f * (W[4 * N + n] * iU0 - 0.5f * (uu * uu + vv * vv + ww * ww));
    const float sd = fsqrt(d_temp);
    const float S = 110.4f / (float)g.P.t_inf;
    g.prim32[LF_MU * N + n] = (sd * sd * sd) * qdiv(1.0f + S, d_temp + S);
}

// Faces along D of one staged tile (face_tile.cuh): the block of
// kFaceThreads threads stages the tile's stencil lines into smem
// (tile_smem_floats<T>() floats) and each thread evaluates its face.  Every
// thread of the block must call it (it synchronises the block).
template <class T, int D>
__device__ __forceinline__ void face_tile(const LatView &g, TileAt at, float *smem)
{
    constexpr int S = T::kStaged;
    float *sQ = smem, *sR = smem + 5 * S, *sF = smem + 10 * S;
    const int N = g.N;
    int n, t, a;
    const bool face = tile_face<T, D>(g, at, n, t, a);
    stage_face_lines<T, D>(g, at, sQ, sR, sF);
    if (!face) return;
    float m[3];   // loaded here: before the staging it costs registers (a direction along k 0.072 -> 0.082 ms)
#pragma unroll
    for (int c = 0; c < 3; ++c) m[c] = lat_ldg(g.fm32 + (size_t)(D * 3 + c) * N, 4u * n);
    const float det_f = lat_ldg(g.fdet32 + (size_t)D * N, 4u * n);
    float2 P[3][5];
    float r[5];
    tile_stencil<T>(sQ, sR, t, a, P, r);
    float Fhat[5];
    x2::llf_face_flux2(P, m[0], m[1], m[2], det_f, r, x2::weno_eps2(g.P), Fhat);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        float f[6];
        tile_node_fluxes<T>(sF, q, t, a, f);
        lat_at(g.Fh32, D * 5 + q, N, n) = __fadd_rn(Fhat[q], x2::face_correction_sym(f));
    }
}

// RHS and SSP-RK3 stage jst from the FP32 face and viscous fluxes, then the
// next stage's U_Q.  L is summed in FP32 (neighbouring face fluxes within a
// factor of two subtract exactly); the RK accumulation is hi/lo:
//   jst 0: U1 = U0 + dt L
//   jst 1: U2 = 3/4 U0 + 1/4 U1 + 1/4 dt L
//   jst 2: U0 = (U0 + 2 (U2 + dt L)) / 3
// and the new state lands in slot (jst+1) mod 3, which is also the next
// stage's U_Q slot.  LOC as for visc_node.
template <bool LOC>
__device__ __forceinline__ void update_node(const LatView &g, int n, int jst)
{
    const int N = g.N;
    if (LOC && lat_ghost(g, n)) {
        // Ghosts are the boundary routine's, which fills those next to face
        // nodes after this kernel; the others (behind edges and corners) keep
        // their state, which moves on to the next stage's slot.
        if (g.Lout) {
#pragma unroll
            for (int c = 0; c < 5; ++c) g.Lout[c * N + n] = 0.0;
        }
        dfl Us[5];
        load_state(g, jst, n, Us);
        store_state(g, jst == 2 ? 0 : jst + 1, n, Us);
        return;
    }
    int i, j, k;
    lat_ijk(g, n, i, j, k);
    const unsigned lflag = (LOC && g.locflag) ? g.locflag[n] : 7u;
    float Lf[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int m1 = lat_step(g, i, j, k, d, -1);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const float *Fd = g.Fh32 + (size_t)(d * 5 + c) * N;
            Lf[c] += lat_ldg(Fd, 4u * n) - lat_ldg(Fd, 4u * m1);
        }
        if (LOC && g.P.viscous && lat_locdir(g, d) && ((lflag >> d) & 1u)) {
            int s[7], L7[7];
#pragma unroll
            for (int o = 0; o < 7; ++o) {
                s[o] = lat_step(g, i, j, k, d, o - 3);
                L7[o] = g.loc8[s[o]];
            }
            const int b = weno_visc_branch(L7);
            const float *Vd = g.V32 + (size_t)d * 5 * N;
#pragma unroll
            for (int c = 1; c < 5; ++c) {
                float f[7];
#pragma unroll
                for (int o = 0; o < 7; ++o) f[o] = __ldg(Vd + c * N + s[o]);
                Lf[c] += branch_deriv<float>(b, f);
            }
        } else if (g.P.viscous) {
            const int m2 = lat_step(g, i, j, k, d, -2), p1 = lat_step(g, i, j, k, d, 1), p2 = lat_step(g, i, j, k, d, 2);
#pragma unroll
            for (int c = 1; c < 5; ++c) {
                const float *V = g.V32 + (size_t)(d * 5 + c) * N;
                const float d1 = lat_ldg(V, 4u * p1) - lat_ldg(V, 4u * m1),
                            d2 = lat_ldg(V, 4u * p2) - lat_ldg(V, 4u * m2);
                Lf[c] = fmaf(1.0f / 12.0f, fmaf(8.0f, d1, -d2), Lf[c]);
            }
        }
    }
    if (g.Lout) {
#pragma unroll
        for (int c = 0; c < 5; ++c) g.Lout[c * N + n] = -(double)Lf[c];
    }
    const dfl dt = {g.dt_hi, g.dt_lo};
    dfl U0[5], Un[5];
    load_state(g, 0, n, U0);
    if (jst == 0) {
#pragma unroll
        for (int c = 0; c < 5; ++c) Un[c] = df_add(U0[c], df_mul({-Lf[c], 0.0f}, dt));
    } else if (jst == 1) {
        dfl U1[5];
        load_state(g, 1, n, U1);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const dfl a = df_mul(U0[c], {0.75f, 0.0f});
            const dfl b = {0.25f * U1[c].h, 0.25f * U1[c].l};
            const dfl t = df_mul({-0.25f * Lf[c], 0.0f}, dt);
            Un[c] = df_add(df_add(a, b), t);
        }
    } else {
        dfl U2[5];
        load_state(g, 2, n, U2);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const dfl a = df_add(U2[c], df_mul({-Lf[c], 0.0f}, dt));   // (U0 + 2 (U2 + dt L)) / 3
            Un[c] = df_mul(df_add(U0[c], {2.0f * a.h, 2.0f * a.l}), {kThirdH, kThirdL});
        }
    }
    store_state(g, jst == 2 ? 0 : jst + 1, n, Un);
    derive(g, n, Un);
}

// ------------------------------------------------ boundary routine ---

// Target m of one entry of the reference's boundary routine
// (bc_target_rules) on the hi/lo state in slot q.  A node that is written
// takes its state and the next stage's U_Q outputs.
struct HiLoState {
    const LatView &g;
    int q;
    __device__ __forceinline__ double det(int n) const { return g.det[n]; }
    __device__ __forceinline__ void U(int n, double U[5]) const
    {
        const float *W = lat_W(g, q);
#pragma unroll
        for (int c = 0; c < 5; ++c) U[c] = emu::f2d(W[c * g.N + n]) + emu::f2d(W[(5 + c) * g.N + n]);
    }
    __device__ __forceinline__ void put(int n, const double U[5]) const
    {
        dfl Un[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) emu::hi_lo(U[c], Un[c].h, Un[c].l);
        store_state(g, q, n, Un);
        derive(g, n, Un);
    }
    __device__ __forceinline__ void set(int n, double rho, double u, double v, double w, double p) const
    {
        const double D = g.det[n];
        const double E = p / 0.4 + 0.5 * rho * (u * u + v * v + w * w);
        const double U[5] = {D * rho, D * rho * u, D * rho * v, D * rho * w, D * E};
        put(n, U);
    }
};

__device__ __forceinline__ void bc_target(const LatView &g, int type, const BcEntry &e, int m, int q, double mach)
{
    bc_target_rules(HiLoState{g, q}, type, e, m, mach);
}

// FP64 FLOW of a node from its conserved state, the quotients and the root
// on the integer pipe (the same bits): 16 operations of the FP64 pipe, which
// bounds this kernel, where eight quotients and a root took some ninety
// (2.1 million nodes: 0.35 -> 0.11 ms).  SPLIT: e from p as the split
// form states it.  mu from the last viscous pass.
template <bool SPLIT>
__device__ __forceinline__ void flow_out(const LatView &g, int n, double id, const double U[5])
{
    const int N = g.N;
    double fu[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) fu[c] = id * U[c];
    const double rho = fu[0];
    const xi::Divisor over = xi::divisor(rho);
    double v[4] = {fu[1], fu[2], fu[3], fu[4]};
    xi::quot_n(v, over);
    const double e = v[3] - 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    const double p = e * rho * 0.4;
    double r[2] = {p, 1.4 * p};
    xi::quot_n(r, over);
    const double mach = g.P.mach;
    double *F = g.prim9;
    F[LF_RHO * N + n] = rho;
    F[LF_U * N + n] = v[0];
    F[LF_V * N + n] = v[1];
    F[LF_W * N + n] = v[2];
    F[LF_E * N + n] = SPLIT ? xi::divide(p, 0.4 * rho) : e;
    F[LF_P * N + n] = p;
    F[LF_T * N + n] = (1.4 * mach * mach) * r[0];
    F[LF_A * N + n] = xi::root(r[1]);
    F[LF_MU * N + n] = emu::f2d(g.prim32[LF_MU * N + n]);
}

// FP64 FLOW of the hi/lo state in slot q (boundary output).
__device__ __forceinline__ void flow_out_node(const LatView &g, int n, int q)
{
    double U[5];
    HiLoState{g, q}.U(n, U);
    flow_out<false>(g, n, xi::divide(1.0, g.det[n]), U);
}

}  // namespace mx
}  // namespace cfd
