// physics_x2.cuh -- the mixed form's LLF face flux on paired FP32 lanes.
//
// Blackwell issues two FP32 operations per packed instruction (__ffma2_rn,
// __fmul2_rn, __fadd2_rn).  The face flux pairs naturally:
//   * the characteristic projection of stencil point k is paired with that
//     of point 5-k;
//   * WENO5's left-biased ("neg") value is its right-biased ("pos") formula
//     applied to the reversed stencil, so lane x (stencil) and lane y
//     (reversed stencil) of one evaluation give pos and neg;
//   * the back-projection, the contravariant fluxes and the LLF split run on
//     the (pos, neg) pair.
// The formulas follow the reference's Weno kernel (Weno.cl:337-413 eigen
// system, 1056-1280 WENO5, 2188-2583 back-projection and fluxes, 2859-3058
// LLF and the sixth-order correction); only the lane packing is new.
#pragma once

#include "emu64.cuh"
#include "physics.cuh"

namespace cfd {
namespace x2 {

__device__ __forceinline__ float2 b2(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, b2(-1.0f), a); }
__device__ __forceinline__ float2 swap2(float2 a) { return make_float2(a.y, a.x); }
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(frcp(a.x), frcp(a.y)); }

// WENO5 on both lanes (neg, pos) in differences: the face value less a node's
// value, from the lane's one-sided differences away from the node next to the
// face on its own side: d3 (second to third node), d2 (first to second) and
// (-p, p) (across the face); the fourth is -swap(d2).  The candidates
// (15/8,-5/4,3/8 | 3/8,3/4,-1/8 | -1/8,3/4,3/8) less the own node's value, the
// linear weights 1 : 10 : 5 folded into them and w_k = d_k/(eps+IS_k)^2 with
// IS and eps over 13/12 (eps here is 12/13 of
// the scheme's), which the quotient does not see: 30 paired operations
// where the same reconstruction of five values takes 47, and its rounding
// scales with the variation across the stencil.
// LEFT: less the value of the face's left node on both lanes (one operation
// more), else of the lane's own node.  Where the eigenvectors are applied to
// the offsets alone (the split form) the reference has to be one for both
// sides: the approximate roots and reciprocals make R L the identity to some
// 1e-8 with a mean, and what they make of the deviations then scales the
// jump of the face states with them.  Measured from its own node, each side
// leaves that share of the nodes' whole difference in the jump, a dissipation
// of first order: TGV 32^3, 200 steps, kinetic energy against the FP64 form
// -1.7e-7; -1e-8 to -2e-8 from one reference.
template <bool LEFT>
__device__ __forceinline__ float2 weno5_off2(float2 d3, float2 d2, float p, float eps)
{
    const float2 d1 = make_float2(-p, p), s2 = swap2(d2);
    const float2 t0 = sub2(d3, d2), t1 = sub2(d2, d1), t2 = add2(d1, s2);
    const float2 u0 = fma2(b2(-3.0f), d2, d3), u1 = add2(d1, d2), u2 = fma2(b2(3.0f), d1, s2);
    auto weight = [&](float2 t, float2 u) {
        const float2 e = fma2(t, t, fma2(mul2(b2(3.0f / 13.0f), u), u, b2(eps)));
        return rcp2(mul2(e, e));
    };
    const float2 w0 = weight(t0, u0), w1 = weight(t1, u1), w2 = weight(t2, u2);
    const float2 p0 = fma2(b2(3.0f / 8.0f), d3, mul2(b2(-7.0f / 8.0f), d2));
    const float2 p1 = fma2(b2(-30.0f / 8.0f), d1, mul2(b2(-10.0f / 8.0f), d2));
    const float2 p2 = fma2(b2(-25.0f / 8.0f), d1, mul2(b2(-5.0f / 8.0f), s2));
    const float2 den = fma2(b2(10.0f), w1, fma2(b2(5.0f), w2, w0));
    float2 num = fma2(w0, p0, fma2(w1, p1, mul2(w2, p2)));
    if (LEFT) num = fma2(make_float2(0.0f, p), den, num);
    return mul2(num, rcp2(den));
}

// eps of weno5_off2 (FP64 -> FP32 on the integer pipe)
__device__ __forceinline__ float weno_eps2(const Phys &P) { return __fmul_rn(12.0f / 13.0f, emu::d2f(P.eps)); }

// s a + b and s a of a scalar and paired or single values
__device__ __forceinline__ float2 sfma(float s, float2 a, float2 b) { return fma2(b2(s), a, b); }
__device__ __forceinline__ float sfma(float s, float a, float b) { return fmaf(s, a, b); }
__device__ __forceinline__ float2 smul(float s, float2 a) { return mul2(b2(s), a); }
__device__ __forceinline__ float smul(float s, float a) { return __fmul_rn(s, a); }

// r = L d (left eigenvectors of the face, Weno.cl:384-412) by what the rows
// share: the momentum less the Roe velocity times the density, w, its normal
// part and the pressure-like 0.4 dp.  23 operations where the matrix takes
// 25 and some 60 more to set up (right_times2 alike): a direction of TGV
// 128^3, mixed 0.078 -> 0.070 ms, split 0.097 -> 0.091.
template <class V>
__device__ __forceinline__ void left_times(const FaceEigen &f, const V d[5], V r[5])
{
    const V w1 = sfma(-f.ru, d[0], d[1]), w2 = sfma(-f.rv, d[0], d[2]), w3 = sfma(-f.rw, d[0], d[3]);
    const V dp = sfma(f.h2, d[0], sfma(-f.ru, d[1], sfma(-f.rv, d[2], sfma(-f.rw, d[3], d[4]))));
    const V S = sfma(-f.g2, dp, d[0]), e = smul(f.b4, dp);
    const V kw = sfma(f.kx, w1, sfma(f.ky, w2, smul(f.kz, w3)));
    r[0] = sfma(f.kx, S, sfma(f.iz, w2, smul(-f.iy, w3)));
    r[1] = sfma(f.ky, S, sfma(f.ix, w3, smul(-f.iz, w1)));
    r[2] = sfma(f.kz, S, sfma(f.iy, w1, smul(-f.ix, w2)));
    r[3] = sfma(f.ba, kw, e);
    r[4] = sfma(-f.ba, kw, e);
}

// q = R c on both lanes (right eigenvectors of the face, Weno.cl:349-380):
// x = the momentum less the Roe velocity times the density q0.  Mixed form,
// TGV 64^3 after 200 steps, u against the FP64 form: 5.6e-6 with E summed up
// from its largest term, 4.3e-6 to it (4.6e-6 with the matrices).
__device__ __forceinline__ void right_times2(const FaceEigen &f, const float2 c[5], float2 q[5])
{
    const float2 s34 = add2(c[3], c[4]), z = smul(f.ala, sub2(c[3], c[4]));
    const float2 q0 = sfma(f.kx, c[0], sfma(f.ky, c[1], sfma(f.kz, c[2], smul(f.al, s34))));
    const float2 x1 = sfma(f.kx, z, sfma(f.ny, c[2], smul(-f.nz, c[1])));
    const float2 x2 = sfma(f.ky, z, sfma(f.nz, c[0], smul(-f.nx, c[2])));
    const float2 x3 = sfma(f.kz, z, sfma(f.nx, c[1], smul(-f.ny, c[0])));
    q[0] = q0;
    q[1] = sfma(f.ru, q0, x1);
    q[2] = sfma(f.rv, q0, x2);
    q[3] = sfma(f.rw, q0, x3);
    // the large term last: one rounding at the size of E instead of five, which
    // the pressure would take over (below)
    q[4] = sfma(f.ae, s34, sfma(f.h2, q0, sfma(f.ru, x1, sfma(f.rv, x2, smul(f.rw, x3)))));
}

// Contravariant Euler flux of the face states on both lanes through the face
// metric (mx,my,mz) and lambda_5 = U.m + c|m| (Weno.cl:2291-2583).
__device__ __forceinline__ float2 contravariant_flux2(const float2 q[5], float mx, float my, float mz, float2 f[5])
{
    const float2 ir = rcp2(q[0]);
    const float2 u = mul2(q[1], ir), v = mul2(q[2], ir), w = mul2(q[3], ir);
    const float2 ke2 = fma2(q[1], u, fma2(q[2], v, mul2(q[3], w)));        // |m|^2 / rho
    const float2 pr = mul2(b2(0.4f), fma2(b2(-0.5f), ke2, q[4]));
    const float2 hq = fma2(b2(1.4f), q[4], mul2(b2(-0.2f), ke2));
    const float2 un = fma2(b2(mx), u, fma2(b2(my), v, mul2(b2(mz), w)));
    f[0] = mul2(q[0], un);
    f[1] = fma2(q[1], un, mul2(b2(mx), pr));
    f[2] = fma2(q[2], un, mul2(b2(my), pr));
    f[3] = fma2(q[3], un, mul2(b2(mz), pr));
    f[4] = mul2(hq, un);
    const float2 e = fma2(q[4], ir, mul2(b2(-0.5f), fma2(u, u, fma2(v, v, mul2(w, w)))));
    const float2 c2k = mul2(b2(__fmul_rn(1.4f * 0.4f, dot3(mx, mx, my, my, mz, mz))), e);
    return add2(un, make_float2(fsqrt(c2k.x), fsqrt(c2k.y)));
}

// Reconstructed face states of one face on the two lanes, (neg, pos):
// the Roe eigen-system of the face, the characteristic projection, WENO5 on
// both sides and the back-projection (Weno.cl:337-413, 1056-2289).
// P[k][c] = (Q_c of stencil point k, Q_c of point 5-k), k = 0..2, points
// left-2 .. right+2; roe = Roe state of the face; eps = 12/13 of the
// scheme's.  DEV projects the differences between neighbouring points
// instead of the points: the projection is linear and WENO5 is unchanged by
// a constant shift, so the state is the left node's plus R times the
// reconstructed offset; five projections instead of six, a rounding that
// scales with the variation across the stencil instead of with Q, and a
// uniform stencil returns its value exactly.  A direction of TGV 128^3,
// five-value reconstruction against this one: mixed 0.084 -> 0.080 ms,
// split 0.107 -> 0.100.
template <bool DEV>
__device__ __forceinline__ void reconstruct_face2(const float2 P[3][5], float mx, float my, float mz,
                                                  const float roe[5], float eps, float2 q[5])
{
    FaceEigen eg;
    eg.init(mx, my, mz, roe);
    float2 C[5];   // (neg, pos) of each characteristic variable
    if (DEV) {
        float2 D3[5], D2[5];
        float D1[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            D3[c] = sub2(P[0][c], P[1][c]);
            D2[c] = sub2(P[1][c], P[2][c]);
            D1[c] = P[2][c].y - P[2][c].x;
        }
        float2 d3[5], d2[5];
        float d1[5];
        left_times(eg, D3, d3);
        left_times(eg, D2, d2);
        left_times(eg, D1, d1);
#pragma unroll
        for (int r = 0; r < 5; ++r) C[r] = weno5_off2<true>(d3[r], d2[r], d1[r], eps);
    } else {
        float2 c0[5], c1[5], c2[5];
        left_times(eg, P[0], c0);
        left_times(eg, P[1], c1);
        left_times(eg, P[2], c2);
#pragma unroll
        for (int r = 0; r < 5; ++r)
            C[r] = add2(c2[r], weno5_off2<false>(sub2(c0[r], c1[r]), sub2(c1[r], c2[r]), c2[r].y - c2[r].x, eps));
    }
    right_times2(eg, C, q);
    if (DEV) {
#pragma unroll
        for (int c = 0; c < 5; ++c) q[c] = add2(q[c], b2(P[2][c].x));
    }
}

// LLF face flux (Weno.cl:2859-2947): Fhat = 0.5 det (Fp + Fn - alpha (qp - qn)),
// alpha = max |lambda_5|, all FP32.
__device__ __forceinline__ void llf_face_flux2(const float2 P[3][5], float mx, float my, float mz, float det_f,
                                               const float roe[5], float eps, float Fhat[5])
{
    float2 q[5], f[5];
    reconstruct_face2<false>(P, mx, my, mz, roe, eps, q);
    const float2 lam = contravariant_flux2(q, mx, my, mz, f);
    const float alpha = fmaxf(fabsf(lam.x), fabsf(lam.y));
    const float2 sa = make_float2(alpha, -alpha);
    const float hd = 0.5f * det_f;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const float2 t = fma2(sa, q[c], f[c]);
        Fhat[c] = __fmul_rn(hd, t.x + t.y);
    }
}

// The same LLF face flux with the metric and Jacobian products in FP64 (the
// split form): the face states (q+, q-), their velocities and pressures,
// lambda_5 and the dissipation alpha (q+ - q-) in FP32; the
// contravariant fluxes' metric products and their product by det_f / 2 in
// FP64 (Weno.cl:2585-2728, 2913-2947).  The central sum of the two states'
// fluxes q U_n + m p (and (E + p) U_n) is taken as
//   q+ U+ + q- U- = (q+ + q-) (U+ + U-) / 2 + (q+ - q-) (U+ - U-) / 2:
// the first term, which carries the metric, in FP64 with U+ + U- = m.(u+ +
// u-) from the FP64 face metric dm; the second, a product of two
// differences across the face, in FP32 with the dissipation.  A uniform
// stencil (q+ = q-) gives exactly the FP64 flux of that state.  m (FP32) is
// the face metric rounded, for the eigenvectors and lambda_5.  extra[c]
// (FP32) is added to component c with the other FP32 terms.
__device__ __forceinline__ void llf_face_flux2_split(const float2 P[3][5], float mx, float my, float mz,
                                                     const double dm[3], double det_f, const float roe[5], float eps,
                                                     const float extra[5], double Fhat[5])
{
    float2 q[5];
    reconstruct_face2<true>(P, mx, my, mz, roe, eps, q);
    const float2 ir = rcp2(q[0]);
    const float2 u = mul2(q[1], ir), v = mul2(q[2], ir), w = mul2(q[3], ir);
    const float2 ke2 = fma2(q[1], u, fma2(q[2], v, mul2(q[3], w)));        // |m|^2 / rho
    const float2 pr = mul2(b2(0.4f), fma2(b2(-0.5f), ke2, q[4]));
    // lambda_5 = U.m + c |m| in FP32 (the LLF speed)
    const float2 un32 = fma2(b2(mx), u, fma2(b2(my), v, mul2(b2(mz), w)));
    const float2 e = fma2(q[4], ir, mul2(b2(-0.5f), fma2(u, u, fma2(v, v, mul2(w, w)))));
    const float2 c2k = mul2(b2(__fmul_rn(1.4f * 0.4f, dot3(mx, mx, my, my, mz, mz))), e);
    const float2 lam = add2(un32, make_float2(fsqrt(c2k.x), fsqrt(c2k.y)));
    const float alpha = fmaxf(fabsf(lam.x), fabsf(lam.y));
    const double hd = 0.5 * det_f;
    const float hd32 = emu::d2f(hd);
    // FP32 terms: extra, less the dissipation, plus the difference term
    // (q+ - q-) (U+ - U-) / 2, all times det_f / 2 where they belong
    const float dun = un32.y - un32.x;
    float qs[5], x[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const float qp = c == 4 ? q[4].y + pr.y : q[c].y, qn = c == 4 ? q[4].x + pr.x : q[c].x;
        qs[c] = qp + qn;
        x[c] = fmaf(hd32, fmaf(__fmul_rn(0.5f, qp - qn), dun, -__fmul_rn(alpha, q[c].y - q[c].x)), extra[c]);
    }
    // FP64: the metric products of the sum term and of the pressure (the
    // FP32 -> FP64 conversions on the integer pipe, emu::f2d: exact)
    using emu::f2d;
    const double hsun = hd * (0.5 * fma(dm[0], f2d(u.x + u.y), fma(dm[1], f2d(v.x + v.y), dm[2] * f2d(w.x + w.y))));
    const double hps = hd * f2d(pr.x + pr.y);
    Fhat[0] = fma(f2d(qs[0]), hsun, f2d(x[0]));
#pragma unroll
    for (int c = 1; c < 4; ++c) Fhat[c] = fma(dm[c - 1], hps, fma(f2d(qs[c]), hsun, f2d(x[c])));
    Fhat[4] = fma(f2d(qs[4]), hsun, f2d(x[4]));
}

// Sixth-order correction of a face flux from the node fluxes f[0..5]
// (Weno.cl:2950-3058): -d2/24 + 7 d4/5760, d2 = (-5,39,-34,-34,39,-5)/48,
// d4 = (1,-3,2,2,-3,1)/2.  Its coefficients are symmetric and sum to zero:
// taken of the differences from the node next to the face on each side, so
// that it rounds with the variation of the flux.
__device__ __forceinline__ float face_correction_sym(const float f[6])
{
    constexpr float a0 = (float)(5.0 / (48.0 * 24.0) + 7.0 / (5760.0 * 2.0));
    constexpr float a1 = (float)(-39.0 / (48.0 * 24.0) - 21.0 / (5760.0 * 2.0));
    const float2 c = make_float2(f[2], f[3]);
    const float2 g0 = sub2(make_float2(f[0], f[5]), c), g1 = sub2(make_float2(f[1], f[4]), c);
    const float2 s = fma2(b2(a0), g0, mul2(b2(a1), g1));
    return __fadd_rn(s.x, s.y);
}

}  // namespace x2
}  // namespace cfd
