// lattice_split.cuh -- per-node operations of the split-precision lattice
// stage: FP64 for what carries the conserved state and the geometry, FP32
// for the flux physics.
//
// FP64: the state U0/U1/U2 ([5][N] doubles, the FP64 form's layout), the
// SSP-RK3 accumulation (Weno.cl:3084-3126), Q = U / det through the FP64
// reciprocal of det (U_Q.cl:112-122), the contravariant face flux
// DET_f (m_f . F) of the reconstructed face states with its LLF central
// average (Weno.cl:2585-2728, 2913-2947; physics_x2.cuh
// llf_face_flux2_split), and the flux difference L (Weno.cl:3060-3082).
// FP32: the Roe average, eigenvectors, characteristic projection, WENO5 (on
// the stencil's differences), back-projection, the
// face states' velocities and pressures, lambda_5 and the LLF dissipation
// alpha (q+ - q-), the viscous and SGS fluxes and their divergence
// (Viscous.cl:439-631, the mixed form's code on a hi + lo FP32 read copy of
// the FP64 state), and the node fluxes with the sixth-order correction
// -d2/24 + 7 d4/5760 they feed (a high-order correction added to the FP64
// face flux).
// Include only from translation units compiled with FMA contraction and
// approximate FP32 division/square root.
#pragma once

#include "boundary.h"
#include "exact_div.cuh"
#include "lattice.cuh"
#include "lattice_mixed.cuh"
#include "physics_x2.cuh"

namespace cfd {
namespace sp {

__device__ __forceinline__ void load_state(const LatView &g, int q, int n, double Un[5])
{
    const int N = g.N;
    const double *U = lat_U(g, q);
#pragma unroll
    for (int c = 0; c < 5; ++c) Un[c] = lat_at(U, c, N, n);
}

__device__ __forceinline__ void store_state(const LatView &g, int q, int n, const double Un[5])
{
    const int N = g.N;
    double *U = lat_U(g, q);
#pragma unroll
    for (int c = 0; c < 5; ++c) lat_at(U, c, N, n) = Un[c];
}

// U_Q of the next stage from the state Un (= det * Q): Q in FP64, rounded
// once to FP32 for the face stage; the Roe inputs (u, v, w, sqrt(rho), H)
// and the pressure in FP32; and the state as
// hi + lo FP32 pairs in g.Whl ([10][N]), a read copy from which the viscous
// pass takes its neighbour differences on the FP32 pipe (the differences of
// hi parts are exact between neighbours within a factor of two).
__device__ __forceinline__ void derive(const LatView &g, int n, const double Un[5])
{
    const int N = g.N;
    // FP32 <-> FP64 conversions, the hi/lo split and the products by 1/det
    // on the integer pipe (emu64.cuh; the same bits as the FP64 pipe's)
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        float h, l;
        emu::hi_lo(Un[c], h, l);
        lat_at(g.Whl, c, N, n) = h;
        lat_at(g.Whl, 5 + c, N, n) = l;
    }
    const double id = lat_at(g.idet64, 0, N, n);
    float q[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) q[c] = emu::d2f(emu::mul(Un[c], id));
    const float rho = q[0];
    const float ir = frcp(rho);
    const float u = __fmul_rn(q[1], ir), v = __fmul_rn(q[2], ir), w = __fmul_rn(q[3], ir);
    const float p = __fmul_rn(0.4f, fmaf(-0.5f, dot3(q[1], u, q[2], v, q[3], w), q[4]));
    lat_at(g.prim32, LF_P, N, n) = p;
    if (!(isfinite(rho) && isfinite(u) && isfinite(v) && isfinite(w) && isfinite(p))) atomicOr(g.flags, 2u);
#pragma unroll
    for (int c = 0; c < 5; ++c) lat_at(g.Q32, c, N, n) = q[c];
    lat_at(g.R32, 0, N, n) = u;
    lat_at(g.R32, 1, N, n) = v;
    lat_at(g.R32, 2, N, n) = w;
    lat_at(g.R32, 3, N, n) = fsqrt(rho);
    lat_at(g.R32, 4, N, n) = __fmul_rn(q[4] + p, ir);   // H = (E + p) / rho
}

// U = det * Q(FLOW) in FP64 (U_Q.cl:112-116) into slot q, then derive.
__device__ __forceinline__ void set_prims(const LatView &g, int q, int n, double rho, double u, double v, double w,
                                          double p)
{
    const double D = g.det[n];
    const double E = xi::divide(p, 0.4) + 0.5 * rho * (u * u + v * v + w * w);
    const double Un[5] = {D * rho, D * rho * u, D * rho * v, D * rho * w, D * E};
    store_state(g, q, n, Un);
    derive(g, n, Un);
}

// U_Q from the FP64 FLOW (after an upload).
__device__ __forceinline__ void init_node(const LatView &g, int n, int q)
{
    const int N = g.N;
    g.prim32[LF_MU * N + n] = emu::d2f(g.prim9[LF_MU * N + n]);
    set_prims(g, q, n, g.prim9[LF_RHO * N + n], g.prim9[LF_U * N + n], g.prim9[LF_V * N + n], g.prim9[LF_W * N + n],
              g.prim9[LF_P * N + n]);
}

// U_Q from the state in slot src, copied to slot dst.
__device__ __forceinline__ void prep_node(const LatView &g, int n, int src, int dst)
{
    double Un[5];
    load_state(g, src, n, Un);
    if (src != dst) store_state(g, dst, n, Un);
    derive(g, n, Un);
}

// The view the mixed form's viscous pass (mx::visc_node, mx::mu_node) reads
// as its hi/lo state: every U slot aliases the read copy g.Whl of the
// current stage's state, which derive wrote.
__host__ __device__ __forceinline__ LatView hilo_view(const LatView &g)
{
    LatView v = g;
    v.U0 = v.U1 = v.U2 = reinterpret_cast<double *>(g.Whl);
    return v;
}

// The FP64 face flux of face n+1/2 along D from its stencil (P, pairs of
// points k and 5-k) and Roe state r, plus corr, the FP32 sixth-order
// correction of each component.
struct FaceMetric {
    double m[3], det;
    float m32[3];
};
template <int D>
__device__ __forceinline__ FaceMetric face_metric(const LatView &g, int n)
{
    const int N = g.N;
    FaceMetric f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        f.m[c] = lat_ldg(g.fm + (size_t)(D * 3 + c) * N, 8u * n);
        f.m32[c] = lat_ldg(g.fm32 + (size_t)(D * 3 + c) * N, 4u * n);
    }
    f.det = lat_ldg(g.fdet + (size_t)D * N, 8u * n);
    return f;
}

__device__ __forceinline__ void face_flux(const LatView &g, const FaceMetric &f, const float2 P[3][5], const float r[5],
                                          const float corr[5], double out[5])
{
    x2::llf_face_flux2_split(P, f.m32[0], f.m32[1], f.m32[2], f.m, f.det, r, x2::weno_eps2(g.P), corr, out);
}

// Faces along D of one staged tile (mx::face_tile with the FP64 face
// flux of face_flux written to Fh).
template <class T, int D>
__device__ __forceinline__ void face_tile(const LatView &g, TileAt at, float *smem)
{
    constexpr int S = T::kStaged;
    float *sQ = smem, *sR = smem + 5 * S, *sF = smem + 10 * S;
    const int N = g.N;
    int n, t, a;
    stage_face_lines<T, D>(g, at, sQ, sR, sF);
    if (!tile_face<T, D>(g, at, n, t, a)) return;
    float2 P[3][5];
    float r[5];
    tile_stencil<T>(sQ, sR, t, a, P, r);
    float corr[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        float f[6];
        tile_node_fluxes<T>(sF, q, t, a, f);
        corr[q] = x2::face_correction_sym(f);
    }
    double Fh[5];
    face_flux(g, face_metric<D>(g, n), P, r, corr, Fh);
#pragma unroll
    for (int q = 0; q < 5; ++q) lat_at(g.Fh, D * 5 + q, N, n) = Fh[q];
}

// RHS and SSP-RK3 stage jst: the face-flux difference in FP64, the viscous
// divergence in FP32 (added in FP64), and the RK accumulation in FP64:
//   jst 0: U1 = U0 + dt L
//   jst 1: U2 = (3 U0 + (U1 + dt L)) / 4
//   jst 2: U0 = (U0 + 2 (U2 + dt L)) / 3
// The new state lands in slot (jst+1) mod 3, which is also the next stage's
// U_Q slot.  LOC as for the mixed form's update_node.
template <bool LOC>
__device__ __forceinline__ void update_node(const LatView &g, int n, int jst)
{
    const int N = g.N;
    if (LOC && lat_ghost(g, n)) {   // ghosts: the state moves on (mixed form's update_node)
        if (g.Lout) {
#pragma unroll
            for (int c = 0; c < 5; ++c) g.Lout[c * N + n] = 0.0;
        }
        double Us[5];
        load_state(g, jst, n, Us);
        store_state(g, jst == 2 ? 0 : jst + 1, n, Us);
        return;
    }
    int i, j, k;
    lat_ijk(g, n, i, j, k);
    const unsigned lflag = (LOC && g.locflag) ? g.locflag[n] : 7u;
    double Ld[5];   // sum of flux differences (= -L), started by the i direction's
    float Lv[5] = {0.f, 0.f, 0.f, 0.f, 0.f};     // viscous divergence; mass has none
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int m1 = lat_step(g, i, j, k, d, -1);
        // FP64 pipe: the integer-pipe add (emu::add) costs more issue than it
        // frees here (TGV 128^3: update 0.23 -> 0.31 ms with one direction)
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const double *Fd = g.Fh + (size_t)(d * 5 + c) * N;
            const double df = lat_ldg(Fd, 8u * n) - lat_ldg(Fd, 8u * m1);
            Ld[c] = d == 0 ? df : Ld[c] + df;
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
                Lv[c] += branch_deriv<float>(b, f);
            }
        } else if (g.P.viscous) {
            const int m2 = lat_step(g, i, j, k, d, -2), p1 = lat_step(g, i, j, k, d, 1), p2 = lat_step(g, i, j, k, d, 2);
#pragma unroll
            for (int c = 1; c < 5; ++c) {
                const float *V = g.V32 + (size_t)(d * 5 + c) * N;
                const float d1 = lat_ldg(V, 4u * p1) - lat_ldg(V, 4u * m1),
                            d2 = lat_ldg(V, 4u * p2) - lat_ldg(V, 4u * m2);
                Lv[c] = fmaf(1.0f / 12.0f, fmaf(8.0f, d1, -d2), Lv[c]);
            }
        }
    }
#pragma unroll
    for (int c = 1; c < 5; ++c) Ld[c] += emu::f2d(Lv[c]);
    if (g.Lout) {
#pragma unroll
        for (int c = 0; c < 5; ++c) g.Lout[c * N + n] = -Ld[c];
    }
    const double dt = g.dt;
    double U0[5], Un[5];
    load_state(g, 0, n, U0);
    if (jst == 0) {
#pragma unroll
        for (int c = 0; c < 5; ++c) Un[c] = fma(-dt, Ld[c], U0[c]);
    } else if (jst == 1) {
        double U1[5];
        load_state(g, 1, n, U1);
#pragma unroll
        for (int c = 0; c < 5; ++c) Un[c] = xdiv::scale2<-2>(fma(3.0, U0[c], fma(-dt, Ld[c], U1[c])));
    } else {
        double U2[5];
        load_state(g, 2, n, U2);
#pragma unroll
        for (int c = 0; c < 5; ++c) Un[c] = emu::mul(1.0 / 3.0, fma(2.0, fma(-dt, Ld[c], U2[c]), U0[c]));
    }
    store_state(g, jst == 2 ? 0 : jst + 1, n, Un);
    derive(g, n, Un);
}

// ------------------------------------------------ boundary routine ---

struct F64State {
    const LatView &g;
    int q;
    __device__ __forceinline__ double det(int n) const { return g.det[n]; }
    __device__ __forceinline__ void U(int n, double U[5]) const { load_state(g, q, n, U); }
    __device__ __forceinline__ void put(int n, const double U[5]) const
    {
        store_state(g, q, n, U);
        derive(g, n, U);
    }
    __device__ __forceinline__ void set(int n, double rho, double u, double v, double w, double p) const
    {
        set_prims(g, q, n, rho, u, v, w, p);
    }
};

__device__ __forceinline__ void bc_target(const LatView &g, int type, const BcEntry &e, int m, int q, double mach)
{
    bc_target_rules(F64State{g, q}, type, e, m, mach);
}

// FP64 FLOW of the state in slot q (boundary output).
__device__ __forceinline__ void flow_out_node(const LatView &g, int n, int q)
{
    double U[5];
    load_state(g, q, n, U);
    mx::flow_out<true>(g, n, g.idet64[n], U);
}

}  // namespace sp
}  // namespace cfd
