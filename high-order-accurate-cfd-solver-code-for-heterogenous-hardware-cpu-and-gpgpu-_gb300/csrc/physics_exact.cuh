// physics_exact.cuh -- FP64 device arithmetic in the reference's own
// evaluation order.
//
// The reference's right-hand side at low Mach number is a small difference
// of large pressure fluxes: re-associating one sum or contracting a*b+c into
// an FMA moves L by 1e-12 .. 1e-11 (relative L2) on the Taylor-Green case.
// The FP64 path therefore evaluates every expression exactly as the
// reference kernels write it (same operand order, same divisions, no
// algebraic rewriting) and the translation units that include this header
// are compiled with --fmad=false.  With IEEE-correct division and square
// root on the GPU this reproduces the reference's results to the last bit
// except where libm functions differ (cbrt).  The products, quotients and
// roots run on the integer pipe (exact_int.cuh; divisions that share a
// divisor share its reciprocal, `Over`), which decides their rounding
// exactly: the same bits, with most of the work moved from the FP64 pipe (two
// operations per clock per SM on GB300).
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "emu64.cuh"
#include "exact_div.cuh"
#include "physics.cuh"

namespace cfd {
namespace ex {

__device__ __forceinline__ double sq(double x) { return x * x; }

// Division of several numerators by one divisor b: Over(b)(x) == x / b, bit
// for bit, with the reciprocal computed once (exact_int.cuh).
struct Over {
    xi::Divisor d;
    __device__ __forceinline__ explicit Over(double divisor) : d(xi::divisor(divisor)) {}
    // with Y of xi::Divisor given as a double's bits (y of reciprocal())
    __device__ __forceinline__ Over(double divisor, double y)
        : d{xi::hi32(y), xi::lo32(y), xi::hi32(divisor), xi::lo32(divisor)}
    {
    }
    __device__ __forceinline__ double reciprocal() const { return xi::words(d.yh, d.yl); }
    __device__ __forceinline__ double operator()(double x) const
    {
        double q[1] = {x};
        xi::quot_n(q, d);
        return q[0];
    }
    template <int N>
    __device__ __forceinline__ void all(double (&x)[N]) const
    {
        xi::quot_n(x, d);
    }
};

// a / b with the same bits (exact_int.cuh).
__device__ __forceinline__ double dv(double a, double b) { return xi::divide(a, b); }

// U_Q.cl:64-65
__device__ __forceinline__ double enthalpy(double rho, double u, double v, double w, double p)
{
    return dv((dv(p, 0.4) + xdiv::scale2<-1>(rho) * (u * u + v * v + w * w) + p), rho);
}

// U_Q.cl:60-109 for one face: {u, v, w, h, rho}; (sb,...) the neighbour.
__device__ __forceinline__ void roe(double sb, double ub, double vb, double wb, double hb, double si, double ui,
                                    double vi, double wi, double hi, double r[5])
{
    r[4] = sb * si;
    const Over d(sb + si);
    r[0] = d(sb * ub + si * ui);
    r[1] = d(sb * vb + si * vi);
    r[2] = d(sb * wb + si * wi);
    r[3] = d(sb * hb + si * hi);
}

// WENO5 pair, Weno.cl:1056-1280; c[0..5] = left-2 .. right+2.
__device__ __forceinline__ void weno_pair(const double cc[6], double eps, double &pos, double &neg)
{
    const double *c = cc + 2;   // c[0] = left node of the face
    // products by 2, 4, 1/4 and 1/8 on the integer pipe (xdiv::scale2,
    // the same bits as the multiplies)
    using xdiv::scale2;
    const double p0 = (15.0 / 8.0) * c[1] - (5.0 / 4.0) * c[2] + (3.0 / 8.0) * c[3];
    const double p1 = (3.0 / 8.0) * c[0] + (3.0 / 4.0) * c[1] - scale2<-3>(c[2]);
    const double p2 = -scale2<-3>(c[-1]) + (3.0 / 4.0) * c[0] + (3.0 / 8.0) * c[1];
    const double m0 = p1;
    const double m1 = p2;
    const double m2 = (3.0 / 8.0) * c[-2] - (5.0 / 4.0) * c[-1] + (15.0 / 8.0) * c[0];
    const double ISm2 = (13.0 / 12.0) * (sq(c[-2] - scale2<1>(c[-1]) + c[0])) + scale2<-2>(sq(c[-2] - scale2<2>(c[-1]) + 3.0 * c[0]));
    const double ISm1 = (13.0 / 12.0) * (sq(c[-1] - scale2<1>(c[0]) + c[1])) + scale2<-2>(sq(c[-1] - c[1]));
    const double ISm0 = (13.0 / 12.0) * (sq(c[0] - scale2<1>(c[1]) + c[2])) + scale2<-2>(sq(3.0 * c[0] - scale2<2>(c[1]) + c[2]));
    const double ISp2 = (13.0 / 12.0) * (sq(c[-1] - scale2<1>(c[0]) + c[1])) + scale2<-2>(sq(c[-1] - scale2<2>(c[0]) + 3.0 * c[1]));
    const double ISp1 = (13.0 / 12.0) * (sq(c[0] - scale2<1>(c[1]) + c[2])) + scale2<-2>(sq(c[0] - c[2]));
    const double ISp0 = (13.0 / 12.0) * (sq(c[1] - scale2<1>(c[2]) + c[3])) + scale2<-2>(sq(3.0 * c[1] - scale2<2>(c[2]) + c[3]));
    const double wp0 = dv(1.0 / 16.0, sq(eps + (ISp0)));
    const double wp1 = dv(5.0 / 8.0, sq(eps + (ISp1)));
    const double wp2 = dv(5.0 / 16.0, sq(eps + (ISp2)));
    const double wm0 = dv(5.0 / 16.0, sq(eps + (ISm0)));
    const double wm1 = dv(5.0 / 8.0, sq(eps + (ISm1)));
    const double wm2 = dv(1.0 / 16.0, sq(eps + (ISm2)));
    const Over sp(wp0 + wp1 + wp2), sm(wm0 + wm1 + wm2);
    const double Wp0 = sp(wp0), Wp1 = sp(wp1), Wp2 = sp(wp2);
    const double Wm0 = sm(wm0), Wm1 = sm(wm1), Wm2 = sm(wm2);
    pos = Wp0 * p0 + Wp1 * p1 + Wp2 * p2;
    neg = Wm0 * m0 + Wm1 * m1 + Wm2 * m2;
}

// The quotients by rho of a face state q (conservative) that its Cartesian
// fluxes and lambda_5 divide by q[0]: q1^2/q0, q2^2/q0, q3^2/q0,
// q1 q2/q0, q1 q3/q0, q2 q3/q0, q1/q0, q2/q0, q3/q0, q4/q0.
struct StateQuot {
    double k1, k2, k3, e12, e13, e23, v1, v2, v3, v4;
};

__device__ __forceinline__ StateQuot state_quot(const double q[5])
{
    const Over d(q[0]);
    double a[6] = {q[1] * q[1], q[2] * q[2], q[3] * q[3], q[1] * q[2], q[1] * q[3], q[2] * q[3]};
    double b[4] = {q[1], q[2], q[3], q[4]};
    d.all(a);
    d.all(b);
    return {a[0], a[1], a[2], a[3], a[4], a[5], b[0], b[1], b[2], b[3]};
}

// Cartesian Euler fluxes of a face state, Weno.cl:2291-2507.
__device__ __forceinline__ void cart_flux(const double q[5], const StateQuot &t, double F[5], double E[5], double G[5])
{
    const double k1 = t.k1, k2 = t.k2, k3 = t.k3;
    const double pr = 0.4 * (q[4] - xdiv::scale2<-1>(k1 + k2 + k3));
    const double hq = (1.4 * q[4] - 0.2 * (k1 + k2 + k3));
    F[0] = q[1];
    F[1] = k1 + pr;
    F[2] = t.e12;
    F[3] = t.e13;
    F[4] = hq * t.v1;
    E[0] = q[2];
    E[1] = t.e12;
    E[2] = k2 + pr;
    E[3] = t.e23;
    E[4] = hq * t.v2;
    G[0] = q[3];
    G[1] = t.e13;
    G[2] = t.e23;
    G[3] = k3 + pr;
    G[4] = hq * t.v3;
}

// lambda_5 of a face state, Weno.cl:2511-2583 element [4].
__device__ __forceinline__ double lambda5(const double q[5], const StateQuot &t, double mx, double my, double mz)
{
    return (mx * t.v1 + my * t.v2 + mz * t.v3)
           + sqrt(1.4 * 0.4 * (t.v4 - dv(q[1] * q[1] + q[2] * q[2] + q[3] * q[3], xdiv::scale2<1>(q[0] * q[0])))
                  * (mx * mx + my * my + mz * mz));
}

// LLF face flux of one face (Weno.cl:336-2947): Roe eigenvectors from the
// face metric and Roe state r = {u,v,w,h,rho}, projection of the six stencil
// points pts (left-2 .. right+2), WENO5, back-projection, contravariant
// fluxes x face det, lambda_5 LLF.
__device__ __forceinline__ void face_flux(const double pts[6][5], double mx, double my, double mz, double DET_F,
                                          const double r[5], double eps, double Fhat[5])
{
    const double ru = r[0], rv = r[1], rw = r[2], rh = r[3], rrho = r[4];
    const double kk = sqrt(mx * mx + my * my + mz * mz);
    const double a = sqrt(0.4 * (rh - xdiv::scale2<-1>(ru * ru + rv * rv + rw * rw)));
    const Over dk(kk);
    const double kx = dk(mx), ky = dk(my), kz = dk(mz);
    const double theta = kx * ru + ky * rv + kz * rw;
    const double phi_sq = 0.5 * 0.4 * (ru * ru + rv * rv + rw * rw);
    const double alpha = dv(rrho, sqrt(2.0) * a);
    const double beta = dv(1.0, sqrt(2.0) * rrho * a);
    double cpos[5], cneg[5];
    {
        const Over da(a * a), dr(rrho);
        const double f = da(phi_sq);
        const double Lm[5][5] = {
            {kx * (1.0 - f) - dr(kz * rv - ky * rw), da(kx * 0.4 * ru), da(kx * 0.4 * rv) + dr(kz),
             da(kx * 0.4 * rw) - dr(ky), da(-kx * 0.4)},
            {ky * (1.0 - f) - dr(kx * rw - kz * ru), da(ky * 0.4 * ru) - dr(kz), da(ky * 0.4 * rv),
             da(ky * 0.4 * rw) + dr(kx), da(-ky * 0.4)},
            {kz * (1.0 - f) - dr(ky * ru - kx * rv), da(kz * 0.4 * ru) + dr(ky), da(kz * 0.4 * rv) - dr(kx),
             da(kz * 0.4 * rw), da(-kz * 0.4)},
            {beta * (phi_sq - theta * a), -beta * (0.4 * ru - kx * a), -beta * (0.4 * rv - ky * a),
             -beta * (0.4 * rw - kz * a), beta * 0.4},
            {beta * (phi_sq + theta * a), -beta * (0.4 * ru + kx * a), -beta * (0.4 * rv + ky * a),
             -beta * (0.4 * rw + kz * a), beta * 0.4}};
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            double cv[6];
#pragma unroll
            for (int o = 0; o < 6; ++o)
                cv[o] = Lm[q][0] * pts[o][0] + Lm[q][1] * pts[o][1] + Lm[q][2] * pts[o][2] + Lm[q][3] * pts[o][3]
                        + Lm[q][4] * pts[o][4];
            weno_pair(cv, eps, cpos[q], cneg[q]);
        }
    }
    double qp[5], qn[5];
    {
        const Over d4(0.4);
        const double R[5][5] = {
            {kx, ky, kz, alpha, alpha},
            {kx * ru, ky * ru - kz * rrho, kz * ru + ky * rrho, alpha * (ru + kx * a), alpha * (ru - kx * a)},
            {kx * rv + kz * rrho, ky * rv, kz * rv - kx * rrho, alpha * (rv + ky * a), alpha * (rv - ky * a)},
            {kx * rw - ky * rrho, ky * rw + kx * rrho, kz * rw, alpha * (rw + kz * a), alpha * (rw - kz * a)},
            {d4(kx * phi_sq) + rrho * (kz * rv - ky * rw), d4(ky * phi_sq) + rrho * (kx * rw - kz * ru),
             d4(kz * phi_sq) + rrho * (ky * ru - kx * rv), alpha * (d4(phi_sq + a * a) + theta * a),
             alpha * (d4(phi_sq + a * a) - theta * a)}};
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            qp[q] = R[q][0] * (cpos[0]) + R[q][1] * (cpos[1]) + R[q][2] * (cpos[2]) + R[q][3] * (cpos[3])
                    + R[q][4] * (cpos[4]);
            qn[q] = R[q][0] * (cneg[0]) + R[q][1] * (cneg[1]) + R[q][2] * (cneg[2]) + R[q][3] * (cneg[3])
                    + R[q][4] * (cneg[4]);
        }
    }
    const StateQuot tp = state_quot(qp), tn = state_quot(qn);
    const double lp = lambda5(qp, tp, mx, my, mz);
    const double ln = lambda5(qn, tn, mx, my, mz);
    double al = __longlong_as_double(0x7ff8000000000000ULL);   // NaN when neither branch holds (NaN input)
    if (fabs(lp) >= fabs(ln)) al = fabs(lp);
    else if (fabs(ln) >= fabs(lp)) al = fabs(ln);
    double Fp[5], Ep[5], Gp[5];
    cart_flux(qp, tp, Fp, Ep, Gp);
    double Fn[5], En[5], Gn[5];
    cart_flux(qn, tn, Fn, En, Gn);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const double fcp = DET_F * (mx * Fp[c] + my * Ep[c] + mz * Gp[c]);
        const double fcn = DET_F * (mx * Fn[c] + my * En[c] + mz * Gn[c]);
        const double qpd = DET_F * qp[c], qnd = DET_F * qn[c];
        Fhat[c] = xdiv::scale2<-1>(fcp + fcn - al * (qpd - qnd));
    }
}

// ------------------------------------------------ the face flux in parts --
// face_flux above in three parts that run as kernels of their own, the same
// expressions in the same order (the same bits): the Roe state's scalars
// (face_base), one characteristic field's projection and WENO5 pair
// (char_pair), and everything after it (flux_from_char).

// Scalars of one face's Roe state that its eigenvectors are built from.
enum { FB_U, FB_V, FB_W, FB_R, FB_A, FB_TH, FB_PHI, FB_OMF, FB_ALPHA, FB_BETA, FB_YA2, FB_YR, FB_N };

// Unit normal of a face metric (Weno.cl:337-348).
__device__ __forceinline__ void face_normal(double mx, double my, double mz, double k[3])
{
    const Over dk(sqrt(mx * mx + my * my + mz * mz));
    double q[3] = {mx, my, mz};
    dk.all(q);
    k[0] = q[0];
    k[1] = q[1];
    k[2] = q[2];
}

// r = {u, v, w, h, rho} of the face, k its unit normal.
__device__ __forceinline__ void face_base(const double r[5], const double k[3], double B[FB_N])
{
    const double ru = r[0], rv = r[1], rw = r[2], rh = r[3], rrho = r[4];
    const double q2 = ru * ru + rv * rv + rw * rw;
    const double a = xi::root(0.4 * (rh - xdiv::scale2<-1>(q2)));
    const double phi_sq = 0.5 * 0.4 * q2;
    const Over da(a * a), dr(rrho);
    B[FB_U] = ru;
    B[FB_V] = rv;
    B[FB_W] = rw;
    B[FB_R] = rrho;
    B[FB_A] = a;
    B[FB_TH] = k[0] * ru + k[1] * rv + k[2] * rw;
    B[FB_PHI] = phi_sq;
    B[FB_OMF] = 1.0 - da(phi_sq);
    double ab[2] = {rrho, 1.0};
    const double by[2] = {sqrt(2.0) * a, sqrt(2.0) * rrho * a};
    xi::div_n(ab, by);
    B[FB_ALPHA] = ab[0];
    B[FB_BETA] = ab[1];
    B[FB_YA2] = da.reciprocal();
    B[FB_YR] = dr.reciprocal();
}

// Row q of the left eigenvectors (Weno.cl:384-412).  Rows 0..2 are one
// expression with x, y, z turned: velocity component c = q and the two that
// follow it cyclically.  base(s) and kn(c) read a scalar of face_base and a
// component of the normal (from memory, so that the turned order costs
// nothing).
template <class Base, class Normal>
__device__ __forceinline__ void left_row(int q, const Base &base, const Normal &kn, double L[5])
{
    if (q < 3) {
        const int n = q == 2 ? 0 : q + 1, m = q == 0 ? 2 : q - 1;
        const double kc = kn(q), kq = kn(n), km = kn(m);
        const double rc = base(FB_U + q), rq = base(FB_U + n), rm = base(FB_U + m);
        const double a = base(FB_A);
        const Over da(a * a, base(FB_YA2)), dr(base(FB_R), base(FB_YR));
        const double kc4 = kc * 0.4;
        double x[4] = {kc4 * rc, kc4 * rq, kc4 * rm, kc4}, y[3] = {km * rq - kq * rm, km, kq};
        da.all(x);
        dr.all(y);
        L[0] = kc * base(FB_OMF) - y[0];
        const double lc = x[0], lq = x[1] + y[1], lm = x[2] - y[2];
        L[1] = q == 0 ? lc : (q == 1 ? lm : lq);
        L[2] = q == 0 ? lq : (q == 1 ? lc : lm);
        L[3] = q == 0 ? lm : (q == 1 ? lq : lc);
        L[4] = -x[3];
    } else {
        const double a = base(FB_A), beta = base(FB_BETA);
        const double ta = base(FB_TH) * a;
        L[0] = beta * (base(FB_PHI) + (q == 3 ? -ta : ta));
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double ka = kn(c) * a;
            L[1 + c] = -beta * (0.4 * base(FB_U + c) + (q == 3 ? -ka : ka));
        }
        L[4] = beta * 0.4;
    }
}

// The constant products of one WENO5 pair on the integer pipe: with c0, c1
// the nodes of the face, 3 c, 3/4 c and 3/8 c (one rounding of the
// significand times 3, the others its exponent moved) and 15/8 c of both,
// 5/4 of the next and 3/8 of the outermost nodes.
struct WenoConst {
    double b0, q0, h0, f0, b1, q1, h1, f1, v2, h3, vm1, hm2;
};

__device__ __forceinline__ WenoConst weno_const(double cm2, double cm1, double c0, double c1, double c2, double c3)
{
    WenoConst w;
    uint32_t h[8], l[8], k[8];
    k[0] = xi::small_words<3, 0>(c0, h[0], l[0]);
    k[1] = xi::small_words<15, -3>(c0, h[1], l[1]);
    k[2] = xi::small_words<3, 0>(c1, h[2], l[2]);
    k[3] = xi::small_words<15, -3>(c1, h[3], l[3]);
    k[4] = xi::small_words<5, -2>(c2, h[4], l[4]);
    k[5] = xi::small_words<3, -3>(c3, h[5], l[5]);
    k[6] = xi::small_words<5, -2>(cm1, h[6], l[6]);
    k[7] = xi::small_words<3, -3>(cm2, h[7], l[7]);
    w.b0 = xi::words(h[0], l[0]);
    w.q0 = xi::words(h[0] - (2u << 20), l[0]);
    w.h0 = xi::words(h[0] - (3u << 20), l[0]);
    w.f0 = xi::words(h[1], l[1]);
    w.b1 = xi::words(h[2], l[2]);
    w.q1 = xi::words(h[2] - (2u << 20), l[2]);
    w.h1 = xi::words(h[2] - (3u << 20), l[2]);
    w.f1 = xi::words(h[3], l[3]);
    w.v2 = xi::words(h[4], l[4]);
    w.h3 = xi::words(h[5], l[5]);
    w.vm1 = xi::words(h[6], l[6]);
    w.hm2 = xi::words(h[7], l[7]);
    if (__builtin_expect((k[0] | k[2] | k[4] | k[5] | k[6] | k[7]) != 0u, 0)) {
        w.b0 = xi::small_or(k[0], h[0], l[0], c0, 3.0);
        w.q0 = xi::small_or(k[0], h[0] - (2u << 20), l[0], c0, 3.0 / 4.0);
        w.h0 = xi::small_or(k[0], h[0] - (3u << 20), l[0], c0, 3.0 / 8.0);
        w.f0 = xi::small_or(k[1], h[1], l[1], c0, 15.0 / 8.0);
        w.b1 = xi::small_or(k[2], h[2], l[2], c1, 3.0);
        w.q1 = xi::small_or(k[2], h[2] - (2u << 20), l[2], c1, 3.0 / 4.0);
        w.h1 = xi::small_or(k[2], h[2] - (3u << 20), l[2], c1, 3.0 / 8.0);
        w.f1 = xi::small_or(k[3], h[3], l[3], c1, 15.0 / 8.0);
        w.v2 = xi::small_or(k[4], h[4], l[4], c2, 5.0 / 4.0);
        w.h3 = xi::small_or(k[5], h[5], l[5], c3, 3.0 / 8.0);
        w.vm1 = xi::small_or(k[6], h[6], l[6], cm1, 5.0 / 4.0);
        w.hm2 = xi::small_or(k[7], h[7], l[7], cm2, 3.0 / 8.0);
    }
    return w;
}

// Called between the phases of one field's reconstruction.  BlockSync keeps
// the warps of a block within a phase, so that they fetch the same few KB of
// its 59 KB of code.  It is a barrier of the whole block: every thread meets
// every one of them, those without a face (`face` false: past the range, or
// a node whose face is not needed) included; only what lies between is theirs
// to skip.
struct NoSync {
    __device__ __forceinline__ void operator()() const {}
};
struct BlockSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

// weno_pair with its products on the integer pipe, from the six projected
// points c, two barriers between its three phases.
template <class Sync = NoSync>
__device__ __forceinline__ void weno_pair_i(bool face, const double c[6], double eps, double &pos, double &neg,
                                            const Sync &sync = Sync())
{
    using xdiv::scale2;
    double p0, p1, p2, m2, S[6];
    if (face) {   // the candidates and the weights' denominators
        const double cm2 = c[0], cm1 = c[1], c0 = c[2], c1 = c[3], c2 = c[4], c3 = c[5];
        const WenoConst kc = weno_const(cm2, cm1, c0, c1, c2, c3);
        p0 = kc.f1 - kc.v2 + kc.h3;
        p1 = kc.h0 + kc.q1 - scale2<-3>(c2);
        p2 = -scale2<-3>(cm1) + kc.q0 + kc.h1;
        m2 = kc.hm2 - kc.vm1 + kc.f0;
        const double b0 = kc.b0, b1 = kc.b1;   // 3 c0, 3 c1
        double T[4] = {cm2 - scale2<1>(cm1) + c0, cm1 - scale2<1>(c0) + c1, c0 - scale2<1>(c1) + c2,
                       c1 - scale2<1>(c2) + c3};
        xi::sq_n(T);
        {
            const xi::Fac k = xi::fac(13.0 / 12.0);
            const xi::Fac a[4] = {k, k, k, k}, b[4] = {xi::fac(T[0]), xi::fac(T[1]), xi::fac(T[2]), xi::fac(T[3])};
            xi::mul_n(a, b, T);
        }
        S[0] = cm2 - scale2<2>(cm1) + b0;
        S[1] = cm1 - c1;
        S[2] = b0 - scale2<2>(c1) + c2;
        S[3] = cm1 - scale2<2>(c0) + b1;
        S[4] = c0 - c2;
        S[5] = b1 - scale2<2>(c2) + c3;
        xi::sq_n(S);
        S[0] = eps + (T[0] + scale2<-2>(S[0]));
        S[1] = eps + (T[1] + scale2<-2>(S[1]));
        S[2] = eps + (T[2] + scale2<-2>(S[2]));
        S[3] = eps + (T[1] + scale2<-2>(S[3]));
        S[4] = eps + (T[2] + scale2<-2>(S[4]));
        S[5] = eps + (T[3] + scale2<-2>(S[5]));
        xi::sq_n(S);
    }
    sync();
    if (face) {   // the weights, in place of their denominators
        double w[6] = {1.0 / 16.0, 5.0 / 8.0, 5.0 / 16.0, 5.0 / 16.0, 5.0 / 8.0, 1.0 / 16.0};
        xi::div_n(w, S);
#pragma unroll
        for (int k = 0; k < 6; ++k) S[k] = w[k];
    }
    sync();
    if (!face) return;   // no barrier follows
    double a[3] = {S[5], S[4], S[3]}, b[3] = {S[2], S[1], S[0]};
    Over(a[0] + a[1] + a[2]).all(a);
    Over(b[0] + b[1] + b[2]).all(b);
    const xi::Fac f[6] = {xi::fac(a[0]), xi::fac(a[1]), xi::fac(a[2]), xi::fac(b[0]), xi::fac(b[1]), xi::fac(b[2])};
    const xi::Fac f1 = xi::fac(p1), f2 = xi::fac(p2);
    const xi::Fac v[6] = {xi::fac(p0), f1, f2, f1, f2, xi::fac(m2)};
    double r[6];
    xi::mul_n(f, v, r);
    pos = r[0] + r[1] + r[2];
    neg = r[3] + r[4] + r[5];
}

// One characteristic field of a face: row L of the left eigenvectors (left(L)
// forms it) times the six stencil points (point(o, c): component c of point
// o, left-2 .. right+2), and the WENO5 pair.  With a BlockSync every thread
// of the block calls it, face or not; without a face neither left nor point
// is called and pos and neg are not set.
template <class Left, class Point, class Sync = NoSync>
__device__ __forceinline__ void char_pair(bool face, const Left &left, const Point &point, double eps, double &pos,
                                          double &neg, const Sync &sync = Sync())
{
    xi::Fac f[5];
    if (face) {
        double L[5];
        left(L);
#pragma unroll
        for (int c = 0; c < 5; ++c) f[c] = xi::fac(L[c]);
    }
    sync();
    double cv[6];
    if (face) {
#pragma unroll
        for (int o = 0; o < 6; ++o) {
            xi::Fac p[5];
            double r[5];
#pragma unroll
            for (int c = 0; c < 5; ++c) p[c] = xi::fac(point(o, c));
            xi::mul_n(f, p, r);
            cv[o] = r[0] + r[1] + r[2] + r[3] + r[4];
        }
    }
    sync();
    weno_pair_i(face, cv, eps, pos, neg, sync);
}

// One side's contravariant flux x det_f (Weno.cl:2291-2507, 2585-2728) and
// lambda_5 (Weno.cl:2511-2583) from its conservative state q; mm = m.m.
__device__ __forceinline__ void side_flux(const double q[5], double mx, double my, double mz, double mm, double DET_F,
                                          double f[5], double &lam)
{
    double a[6], b[5];
    {
        const xi::Fac q0 = xi::fac(q[0]), q1 = xi::fac(q[1]), q2 = xi::fac(q[2]), q3 = xi::fac(q[3]);
        const xi::Fac u[7] = {q1, q2, q3, q1, q1, q2, q0}, v[7] = {q1, q2, q3, q2, q3, q3, q0};
        double r[7];
        xi::mul_n(u, v, r);
        const Over d(q[0]);
        const double k = dv(r[0] + r[1] + r[2], xdiv::scale2<1>(r[6]));
#pragma unroll
        for (int i = 0; i < 6; ++i) a[i] = r[i];
        d.all(a);   // q1^2, q2^2, q3^2, q1 q2, q1 q3, q2 q3 over q0
        double b4[4] = {q[1], q[2], q[3], q[4]};
        d.all(b4);
#pragma unroll
        for (int i = 0; i < 4; ++i) b[i] = b4[i];
        b[4] = k;
    }
    const double kk = a[0] + a[1] + a[2];
    const double pr = 0.4 * (q[4] - xdiv::scale2<-1>(kk));
    const double hq = (1.4 * q[4] - 0.2 * kk);
    const xi::Fac fx = xi::fac(mx), fy = xi::fac(my), fz = xi::fac(mz);
    {
        const xi::Fac h = xi::fac(hq);
        const xi::Fac u[6] = {fx, fy, fz, h, h, h};
        const xi::Fac v[6] = {xi::fac(b[0]), xi::fac(b[1]), xi::fac(b[2]), xi::fac(b[0]), xi::fac(b[1]), xi::fac(b[2])};
        double r[6];
        xi::mul_n(u, v, r);
        lam = (r[0] + r[1] + r[2]) + xi::root(xi::mul(xi::mul(1.4 * 0.4, b[3] - b[4]), mm));
        f[4] = r[3];
        f[0] = r[4];
        f[1] = r[5];   // hq v1, hq v2, hq v3 for now
    }
    const xi::Fac m3[3] = {fx, fy, fz};
    auto dot = [&](double x, double y, double z) {
        const xi::Fac v[3] = {xi::fac(x), xi::fac(y), xi::fac(z)};
        double r[3];
        xi::mul_n(m3, v, r);
        return r[0] + r[1] + r[2];
    };
    f[4] = dot(f[4], f[0], f[1]);
    f[0] = dot(q[1], q[2], q[3]);
    f[1] = dot(a[0] + pr, a[3], a[4]);
    f[2] = dot(a[3], a[1] + pr, a[5]);
    f[3] = dot(a[4], a[5], a[2] + pr);
    const xi::Fac fd = xi::fac(DET_F);
    const xi::Fac d5[5] = {fd, fd, fd, fd, fd};
    const xi::Fac v[5] = {xi::fac(f[0]), xi::fac(f[1]), xi::fac(f[2]), xi::fac(f[3]), xi::fac(f[4])};
    double r[5];
    xi::mul_n(d5, v, r);
#pragma unroll
    for (int c = 0; c < 5; ++c) f[c] = r[c];
}

// Component q of both face states from the characteristic values (row q of
// the right eigenvectors, Weno.cl:349-380, 2188-2289): qp, qn.  cpos(s),
// cneg(s) read the values; base and kn as in left_row, rows 1..3 one
// expression turned.
template <class Base, class Normal, class CharP, class CharN>
__device__ __forceinline__ void back_pair(int q, const Base &base, const Normal &kn, const CharP &cpos,
                                          const CharN &cneg, double &qp, double &qn)
{
    xi::Fac r[5];
    const xi::Fac al = xi::fac(base(FB_ALPHA));
    if (q == 0) {
        r[0] = xi::fac(kn(0));
        r[1] = xi::fac(kn(1));
        r[2] = xi::fac(kn(2));
        r[3] = r[4] = al;
    } else if (q < 4) {
        const int c = q - 1, n = c == 2 ? 0 : c + 1, m = c == 0 ? 2 : c - 1;
        const double rc = base(FB_U + c);
        const xi::Fac kc = xi::fac(kn(c)), kq = xi::fac(kn(n)), km = xi::fac(kn(m)), fr = xi::fac(rc),
                      rr = xi::fac(base(FB_R));
        const xi::Fac u[6] = {kc, kq, km, km, kq, kc}, v[6] = {fr, fr, rr, fr, rr, xi::fac(base(FB_A))};
        double t[6], s[2];
        xi::mul_n(u, v, t);
        const xi::Fac aa[2] = {al, al}, w[2] = {xi::fac(rc + t[5]), xi::fac(rc - t[5])};
        xi::mul_n(aa, w, s);
        const xi::Fac fc = xi::fac(t[0]), fn = xi::fac(t[1] - t[2]), fm = xi::fac(t[3] + t[4]);
        r[0] = c == 0 ? fc : (c == 1 ? fm : fn);
        r[1] = c == 0 ? fn : (c == 1 ? fc : fm);
        r[2] = c == 0 ? fm : (c == 1 ? fn : fc);
        r[3] = xi::fac(s[0]);
        r[4] = xi::fac(s[1]);
    } else {
        const double kx = kn(0), ky = kn(1), kz = kn(2), ru = base(FB_U), rv = base(FB_V), rw = base(FB_W);
        const double a = base(FB_A), phi = base(FB_PHI);
        const xi::Fac fkx = xi::fac(kx), fky = xi::fac(ky), fkz = xi::fac(kz), fu = xi::fac(ru), fv = xi::fac(rv),
                      fw = xi::fac(rw), fp = xi::fac(phi), fa = xi::fac(a);
        double e[4], x[6], y[2], z[5];
        {
            const xi::Fac u[3] = {fkx, fky, fkz}, v[3] = {fp, fp, fp};
            double t[3];
            xi::mul_n(u, v, t);
            const xi::Fac ua[2] = {fa, xi::fac(base(FB_TH))}, va[2] = {fa, fa};
            xi::mul_n(ua, va, y);   // a a, theta a
            e[0] = t[0];
            e[1] = t[1];
            e[2] = t[2];
            e[3] = phi + y[0];
            Over(0.4).all(e);
        }
        {
            const xi::Fac u[6] = {fkz, fky, fkx, fkz, fky, fkx}, v[6] = {fv, fw, fw, fu, fu, fv};
            xi::mul_n(u, v, x);
        }
        const xi::Fac rr = xi::fac(base(FB_R));
        const xi::Fac u[5] = {rr, rr, rr, al, al};
        const xi::Fac v[5] = {xi::fac(x[0] - x[1]), xi::fac(x[2] - x[3]), xi::fac(x[4] - x[5]), xi::fac(e[3] + y[1]),
                              xi::fac(e[3] - y[1])};
        xi::mul_n(u, v, z);
        r[0] = xi::fac(e[0] + z[0]);
        r[1] = xi::fac(e[1] + z[1]);
        r[2] = xi::fac(e[2] + z[2]);
        r[3] = xi::fac(z[3]);
        r[4] = xi::fac(z[4]);
    }
    xi::Fac v[5];
    double t[5];
#pragma unroll
    for (int s = 0; s < 5; ++s) v[s] = xi::fac(cpos(s));
    xi::mul_n(r, v, t);
    qp = t[0] + t[1] + t[2] + t[3] + t[4];
#pragma unroll
    for (int s = 0; s < 5; ++s) v[s] = xi::fac(cneg(s));
    xi::mul_n(r, v, t);
    qn = t[0] + t[1] + t[2] + t[3] + t[4];
}

// The LLF flux of a face (Weno.cl:2859-2947) on two neighbouring lanes, the
// even one with the pos state q, the odd one with the neg state (the whole
// warp calls it): each evaluates its side, then fetches the other's flux,
// state x det_f and lambda_5.  Both lanes return the whole Fhat.
__device__ __forceinline__ void llf_lanes(const double q[5], double mx, double my, double mz, double DET_F,
                                          double Fhat[5])
{
    double f[5], lam;
    side_flux(q, mx, my, mz, mx * mx + my * my + mz * mz, DET_F, f, lam);
    const bool neg = (threadIdx.x & 1) != 0;
    lam = fabs(lam);
    const double other = __shfl_xor_sync(0xffffffffu, lam, 1);
    const double lp = neg ? other : lam, ln = neg ? lam : other;
    double al = __longlong_as_double(0x7ff8000000000000ULL);   // NaN when neither branch holds (NaN input)
    if (lp >= ln) al = lp;
    else if (ln >= lp) al = ln;
    const xi::Fac fd = xi::fac(DET_F), fa = xi::fac(al);
    const xi::Fac d5[5] = {fd, fd, fd, fd, fd}, a5[5] = {fa, fa, fa, fa, fa};
    const xi::Fac v[5] = {xi::fac(q[0]), xi::fac(q[1]), xi::fac(q[2]), xi::fac(q[3]), xi::fac(q[4])};
    double s[5];
    xi::mul_n(d5, v, s);
    xi::Fac w[5];
    double sum[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        sum[c] = f[c] + __shfl_xor_sync(0xffffffffu, f[c], 1);
        const double t = __shfl_xor_sync(0xffffffffu, s[c], 1);
        w[c] = xi::fac((neg ? t : s[c]) - (neg ? s[c] : t));
    }
    xi::mul_n(a5, w, s);
#pragma unroll
    for (int c = 0; c < 5; ++c) Fhat[c] = xdiv::scale2<-1>(sum[c] - s[c]);
}

// The two terms of the sixth-order correction of a face flux (corrected):
// a = d2 / 24 and b = 7 d4 / 5760 from the node fluxes f[0..5].
__device__ __forceinline__ void correction_terms(const double f[6], double &a, double &b)
{
    double p[8];   // 5 f0, 39 f1, 34 f2, 34 f3, 39 f4, 5 f5, 3 f1, 3 f4
    uint32_t h[8], l[8], k[8];
    k[0] = xi::small_words<5, 0>(f[0], h[0], l[0]);
    k[1] = xi::small_words<39, 0>(f[1], h[1], l[1]);
    k[2] = xi::small_words<17, 1>(f[2], h[2], l[2]);
    k[3] = xi::small_words<17, 1>(f[3], h[3], l[3]);
    k[4] = xi::small_words<39, 0>(f[4], h[4], l[4]);
    k[5] = xi::small_words<5, 0>(f[5], h[5], l[5]);
    k[6] = xi::small_words<3, 0>(f[1], h[6], l[6]);
    k[7] = xi::small_words<3, 0>(f[4], h[7], l[7]);
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = xi::words(h[i], l[i]);
    if (__builtin_expect((k[0] | k[1] | k[2] | k[3] | k[4] | k[5]) != 0u, 0)) {
        const double x[8] = {f[0], f[1], f[2], f[3], f[4], f[5], f[1], f[4]};
        const double c[8] = {5.0, 39.0, 34.0, 34.0, 39.0, 5.0, 3.0, 3.0};
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = xi::small_or(k[i], h[i], l[i], x[i], c[i]);
    }
    const double s2 = -p[0] + p[1] - p[2] - p[3] + p[4] - p[5];
    const double d4 = xdiv::scale2<-1>(f[0] - p[6] + xdiv::scale2<1>(f[2]) + xdiv::scale2<1>(f[3]) - p[7] + f[5]);
    const xi::Fac u[2] = {xi::fac(1.0 / 48.0), xi::fac(7.0 / 5760.0)}, v[2] = {xi::fac(s2), xi::fac(d4)};
    double r[2];
    xi::mul_n(u, v, r);
    a = xi::mul(1.0 / 24.0, r[0]);
    b = r[1];
}

// Corrected face flux Fhat - d2/24 + 7 d4/5760, Weno.cl:2950-3058, for the
// face between f[2] and f[3] (f[0..5] = left-2 .. right+2).
__device__ __forceinline__ double corrected(double Fhat, const double f[6])
{
    const double d2 = (1.0 / 48.0) * (-5.0 * f[0] + 39.0 * f[1] - 34.0 * f[2] - 34.0 * f[3] + 39.0 * f[4] - 5.0 * f[5]);
    const double d4 = xdiv::scale2<-1>(f[0] - 3.0 * f[1] + xdiv::scale2<1>(f[2]) + xdiv::scale2<1>(f[3]) - 3.0 * f[4] + f[5]);
    return Fhat - (1.0 / 24.0) * d2 + (7.0 / 5760.0) * d4;
}

// r[i] = a[i] b[i], r[i] = k b[i], x[i] = x[i]^2, a b: on the integer pipe
// (I), or on the FP64 pipe with the same bits.  The per-node kernels are
// built both ways: a few blocks per SM cannot keep the FP64 pipe busy, and
// there the integer form's seven times longer code costs more to fetch than
// it saves (kPlainNodes, internal.h).
template <bool I, int N>
__device__ __forceinline__ void products(const double (&a)[N], const double (&b)[N], double (&r)[N])
{
    if (I) {
        xi::Fac fa[N], fb[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            fa[i] = xi::fac(a[i]);
            fb[i] = xi::fac(b[i]);
        }
        xi::mul_n(fa, fb, r);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) r[i] = a[i] * b[i];
    }
}

template <bool I, int N>
__device__ __forceinline__ void scaled(double k, const double (&b)[N], double (&r)[N])
{
    double a[N];
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = k;
    products<I>(a, b, r);
}

template <bool I, int N>
__device__ __forceinline__ void squares(double (&x)[N])
{
    if (I) {
        xi::sq_n(x);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = x[i] * x[i];
    }
}

template <bool I>
__device__ __forceinline__ double product(double a, double b)
{
    return I ? xi::mul(a, b) : a * b;
}

// Fourth-order central first derivatives (Viscous.cl:325-332 and the loc==0
// branch of Weno.cl:2771-2778) of five values; f(o, c): value c at offset o.
template <bool I, class F>
__device__ __forceinline__ void central4(const F &f, double *out)
{
    double b[5], r[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) b[c] = xdiv::scale2<3>(f(1, c) - f(-1, c)) - (f(2, c) - f(-2, c));   // 8 (...): the exponent moved
    scaled<I>(1.0 / 12.0, b, r);
#pragma unroll
    for (int c = 0; c < 5; ++c) out[c] = r[c];
}

// m . (0, 0, 0) x det as the reference evaluates it: a zero, negative where
// the three products are (every component of m negative) or det is, not
// both; NaN from a component or det that is not finite.
__device__ __forceinline__ double zero_dot(double mx, double my, double mz, double det)
{
    const uint32_t hx = xi::hi32(mx), hy = xi::hi32(my), hz = xi::hi32(mz), hd = xi::hi32(det);
    const uint32_t big = 0x7ff00000u;
    if ((hx & big) == big || (hy & big) == big || (hz & big) == big || (hd & big) == big)
        return det * (mx * 0.0 + my * 0.0 + mz * 0.0);
    return xi::words(((hx & hy & hz) ^ hd) & 0x80000000u, 0u);
}

// 1 / det^(1/3), the filter width the SGS terms take (Viscous.cl:490).
__device__ __forceinline__ double filter_width(double det) { return dv(1.0, cbrt(det)); }

// Cartesian flux vectors tF, tE, tG ([N] components) through the node
// metrics (m(k), k = 0..8), x det: store(d, c, det (m_d . (tF, tE, tG)[c])).
// A loop over the directions: the instruction cache holds it once.
template <bool I, int N, class Metric, class Store>
__device__ __forceinline__ void through_metrics(const Metric &m, double det, const double (&tF)[N],
                                                const double (&tE)[N], const double (&tG)[N], const Store &store)
{
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        const double mx = m(3 * d), my = m(3 * d + 1), mz = m(3 * d + 2);
        double s[N], r[N];
#pragma unroll
        for (int c = 0; c < N; ++c) {
            const double a[3] = {mx, my, mz}, b[3] = {tF[c], tE[c], tG[c]};
            double q[3];
            products<I>(a, b, q);
            s[c] = q[0] + q[1] + q[2];
        }
        scaled<I>(det, s, r);
#pragma unroll
        for (int c = 0; c < N; ++c) store(d, c, r[c]);
    }
}

// Viscous.cl:439-631 at one node, in the reference's order.  dU(d, out):
// the derivatives of U along d; Ui[5], node metrics m(k), det, filter width
// DEL, FLOW primitives (rho,u,v,w,p), the three MTS test-filter differences
// K (roots of the reference's KS).  store(d, c, value) takes the
// contravariant viscous fluxes Fv, Ev, Gv (d = 0, 1, 2); mu_out the viscosity
// (the inviscid node fluxes come from node_flux).  The products run on the
// integer pipe in groups, the sums on the FP64 pipe.  Directions, gradients
// and flux rows are loops with their small arrays in local memory: unrolled,
// one node's 10,000 instructions (160 KB) outgrew the instruction cache
// (TGV 128^3 1.54 -> 1.45 ms; 4,913 nodes 82 -> 61 us, and 32 us with the
// products on the FP64 pipe).
template <bool I, class Deriv, class Metric, class Store>
__device__ __forceinline__ void viscous_node(const Deriv &dU, const double Ui[5], const Metric &m, double DET_I,
                                             double DEL, const double prim[5], const double K[3], const Phys &P,
                                             const Store &store, double &mu_out)
{
    using xdiv::scale2;   // products by powers of two: the exponent moved
    double g[4][3], d_temp;   // derivatives of u, v, w and of the energy term along the directions
    {
        double s[4] = {Ui[0], Ui[1], Ui[2], Ui[3]};
        squares<I>(s);
        double x[5] = {1.0, Ui[1], Ui[2], Ui[3], Ui[4]}, y[7] = {Ui[1], Ui[2], Ui[3], Ui[4], s[1], s[2], s[3]};
        Over(Ui[0]).all(x);   // r0, v1, v2, v3, U4 / U0
        Over(s[0]).all(y);    // a1 .. a4, U1^2, U2^2, U3^2 over U0^2
        d_temp = product<I>(P.c_temp, x[4] - scale2<-1>(y[4] + y[5] + y[6]));
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            double du[5];
            dU(d, du);
            const double f[8] = {x[0], y[0], x[0], y[1], x[0], y[2], x[0], y[3]};
            const double e[8] = {du[1], du[0], du[2], du[0], du[3], du[0], du[4], du[0]};
            double r[8], t[3];
            products<I>(f, e, r);
            const double u = r[0] - r[1], v = r[2] - r[3], w = r[4] - r[5];
            const double fv[3] = {x[1], x[2], x[3]}, gv[3] = {u, v, w};
            products<I>(fv, gv, t);
            g[0][d] = u;
            g[1][d] = v;
            g[2][d] = w;
            g[3][d] = r[6] - r[7] - t[0] - t[1] - t[2];
        }
    }
    double mr, kq;
    {
        const double sd = xi::root(d_temp);
        const double mu = product<I>(product<I>(product<I>(sd, sd), sd), dv(P.st1, d_temp + P.st));
        mu_out = mu;
        double q[2] = {product<I>(mu, 1.4), mu};
        const double by[2] = {P.pr_re, P.reynolds};
        xi::div_n(q, by);
        kq = q[0];
        mr = q[1];
    }
    // gradients along x, y, z of one variable's derivatives (heat x, y, z; ux,
    // vy, wz), and the mixed sums s_xy, s_xz, s_yz (s_zx: s_xz the other way
    // round) in the reference's order.  Pass i takes variable p along x and
    // q along y.
    double gt[3], ux, vy, wz, s_xy, s_xz, s_yz, s_zx;
    {
        double sums[6][2], s_back = 0.0;
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
            const int p = (0x100133 >> (4 * i)) & 15, x = (0x221120 >> (4 * i)) & 15;
            const int q = (0x221203 >> (4 * i)) & 15, y = (0x100201 >> (4 * i)) & 15;
            const double a[6] = {g[p][0], g[p][1], g[p][2], g[q][0], g[q][1], g[q][2]};
            const double b[6] = {m(x), m(3 + x), m(6 + x), m(y), m(3 + y), m(6 + y)};
            double r[6];
            products<I>(a, b, r);
            const double s1 = r[0] + r[1] + r[2];
            if (i < 3) {
                sums[i][1] = r[3] + r[4] + r[5];
                sums[i][0] = s1;
            } else {
                sums[i][0] = s1 + r[3] + r[4] + r[5];
            }
            if (i == 4) s_back = r[3] + r[4] + r[5] + r[0] + r[1] + r[2];
        }
        gt[0] = sums[0][0];
        gt[1] = sums[0][1];
        gt[2] = sums[1][0];
        ux = sums[1][1];
        vy = sums[2][0];
        wz = sums[2][1];
        s_xy = sums[3][0];
        s_xz = sums[4][0];
        s_yz = sums[5][0];
        s_zx = s_back;
    }
    double qz, qe, qx, tauzz, tauee, tauxx, tauze, tauzx, tauex;
    {
        const double g[3] = {ux, vy, wz};
        double t[3], r[6], h[3];
        scaled<I>(2.0 / 3.0, g, t);   // 4/3 x is twice 2/3 x
        const double b[6] = {scale2<1>(t[0]) - t[1] - t[2], scale2<1>(t[1]) - t[0] - t[2],
                             scale2<1>(t[2]) - t[0] - t[1], s_xy, s_xz, s_yz};
        scaled<I>(mr, b, r);
        scaled<I>(-kq, gt, h);
        qz = h[0];
        qe = h[1];
        qx = h[2];
        tauzz = r[0];
        tauee = r[1];
        tauxx = r[2];
        tauze = r[3];
        tauzx = r[4];
        tauex = r[5];
    }
    double TAU_XY = 0, TAU_YZ = 0, TAU_XZ = 0, TAU_XX = 0, TAU_YY = 0, TAU_ZZ = 0;
    double H_X = 0, H_Y = 0, H_Z = 0, D_X = 0, D_Y = 0, D_Z = 0;
    const double u = prim[1], v = prim[2], w = prim[3];
    if (P.les) {
        const double C_MTS = 0.03, C_T = 10.0;
        const double yz = scale2<-1>(s_yz), xy = scale2<-1>(s_xy);
        const double xz = scale2<-1>(s_zx);
        double s[6] = {xy, yz, xz, ux, vy, wz};
        squares<I>(s);
        double E[3];
        if (P.les == 2) {
            // Smagorinsky (no counterpart in the reference): (C_s Delta)^2 |S|,
            // |S| = sqrt(2 S_ij S_ij), Delta = det^(1/3) (the cell size; det is
            // the cell volume), in the reference's SGS terms below
            const double S = sqrt(scale2<1>(s[3] + s[4] + s[5]) + scale2<2>(s[0] + s[1] + s[2]));
            const double ls = P.cs * cbrt(DET_I);
            E[0] = E[1] = E[2] = (ls * ls) * S;
        } else {
            const double mod = xi::root(scale2<1>((s[0] + s[1] + s[2]) + product<I>(2.0 / 3.0, s[3] + s[4] + s[5])));
            double c[3] = {C_MTS, C_MTS, C_MTS}, e[3];
            if (mod != 0.0) {
                const double dm = product<I>(DEL, mod);
                double R[3] = {dm, dm, dm};
                const double by[3] = {K[0], K[1], K[2]};
                xi::div_n(R, by);
                Over(C_T).all(R);
                const double one[3] = {1.0 + R[0], 1.0 + R[1], 1.0 + R[2]};
                xi::div_n(c, one);
            }
            scaled<I>(DEL, c, e);
            const double k[3] = {K[0], K[1], K[2]};
            products<I>(e, k, E);
        }
        double r[3], g[3], tau[6], Q[3];
        scaled<I>(-scale2<1>(Ui[0]), E, r);   // -2.0 * U0_I
        scaled<I>(-P.ck, E, g);
        {
            const double a[6] = {r[0], r[1], r[2], r[0], r[1], r[2]}, b[6] = {xy, yz, xz, ux, vy, wz};
            products<I>(a, b, tau);
            products<I>(g, gt, Q);
        }
        TAU_XY = tau[0];
        TAU_YZ = tau[1];
        TAU_XZ = tau[2];
        TAU_XX = tau[3];
        TAU_YY = tau[4];
        TAU_ZZ = tau[5];
        const double a[9] = {TAU_XX, TAU_XY, TAU_XZ, TAU_XY, TAU_YY, TAU_YZ, TAU_XZ, TAU_YZ, TAU_ZZ};
        const double b[9] = {u, u, u, v, v, v, w, w, w};
        double h[9], D[3];
        products<I>(a, b, h);
        H_X = Q[0] + (h[0] + h[1] + h[2]);
        H_Y = Q[1] + (h[3] + h[4] + h[5]);
        H_Z = Q[2] + (h[6] + h[7] + h[8]);
        scaled<I>(0.4, Q, D);
        D_X = D[0];
        D_Y = D[1];
        D_Z = D[2];
    }
    double e[3];
    {
        const double a[9] = {-u, v, w, -u, v, w, -u, v, w};
        const double b[9] = {tauzz, tauze, tauzx, tauze, tauee, tauex, tauzx, tauex, tauxx};
        double r[9];
        products<I>(a, b, r);
        e[0] = (r[0] - r[1] - r[2]) + qz + H_X + D_X;
        e[1] = (r[3] - r[4] - r[5]) + qe + H_Y + D_Y;
        e[2] = (r[6] - r[7] - r[8]) + qx + H_Z + D_Z;
    }
    const double tF[4] = {-tauzz + TAU_XX, -tauze + TAU_XY, -tauzx + TAU_XZ, e[0]};
    const double tE[4] = {-tauze + TAU_XY, -tauee + TAU_YY, -tauex + TAU_YZ, e[1]};
    const double tG[4] = {-tauzx + TAU_XZ, -tauex + TAU_YZ, -tauxx + TAU_ZZ, e[2]};
#pragma unroll 1
    for (int d = 0; d < 3; ++d) store(d, 0, zero_dot(m(3 * d), m(3 * d + 1), m(3 * d + 2), DET_I));
    through_metrics<I>(m, DET_I, tF, tE, tG, [&](int d, int c, double v) { store(d, c + 1, v); });
}

// Contravariant inviscid node fluxes F, E, G (x det; store(d, c, value)) from
// the primitives (rho,u,v,w,p), Viscous.cl:560-578 and 615-631, with the values U_Q shares
// (U_Q.cl:60-122): Q = {rho, rho u, rho v, rho w, E} and the total enthalpy H.
template <bool I, class Metric, class Store>
__device__ __forceinline__ void node_flux(const double prim[5], const Metric &m, double DET_I, const Store &store,
                                          double Q[5], double &H)
{
    const double rho = prim[0], u = prim[1], v = prim[2], w = prim[3], p = prim[4];
    double s[3] = {u, v, w}, r[3], t[9];
    const double vel[3] = {u, v, w};
    squares<I>(s);
    scaled<I>(rho, vel, r);   // rho u, rho v, rho w
    const double en = dv(p, 0.4) + product<I>(xdiv::scale2<-1>(rho), s[0] + s[1] + s[2]);
    const double Et = en + p;
    H = dv(Et, rho);
    Q[0] = rho;
    Q[1] = r[0];
    Q[2] = r[1];
    Q[3] = r[2];
    Q[4] = en;
    {
        // rho u u, rho v u, rho u w, rho v v, rho v w, rho w w, Et u, Et v, Et w
        const double a[9] = {r[0], r[1], r[0], r[1], r[1], r[2], Et, Et, Et}, b[9] = {u, u, w, v, w, w, u, v, w};
        products<I>(a, b, t);
    }
    const double tF[5] = {r[0], t[0] + p, t[1], t[2], t[6]};
    const double tE[5] = {r[1], t[1], t[3] + p, t[4], t[7]};
    const double tG[5] = {r[2], t[2], t[4], t[5] + p, t[8]};
    through_metrics<I>(m, DET_I, tF, tE, tG, store);
}

// Root of the MTS test filter's velocity-difference square
// (Viscous.cl:493-495) for the velocity component c along its own
// direction.  In radix 2 the root of a rounded square is the magnitude
// itself, unless the square leaves the normal range.
__device__ __forceinline__ double ks_root(double Uc_i, double U0_i, double Uc_m, double U0_m, double Uc_p, double U0_p)
{
    using xdiv::scale2;   // 0.25 * x and 0.5 * x on the integer pipe, same bits
    double q[2] = {Uc_i, scale2<-2>(Uc_m) + scale2<-1>(Uc_i) + scale2<-2>(Uc_p)};
    const double by[2] = {U0_i, scale2<-2>(U0_m) + scale2<-1>(U0_i) + scale2<-2>(U0_p)};
    xi::div_n(q, by);
    const double d = q[0] - q[1];
    const uint32_t e = (xi::hi32(d) >> 20) & 0x7ffu;
    if (__builtin_expect(e - 513u >= 1021u, 0)) return d == 0.0 ? 0.0 : sqrt(d * d);
    return fabs(d);
}

// Sutherland viscosity from U only (Viscous.cl:451-458).
template <bool I>
__device__ __forceinline__ double mu_of(const double Ui[5], const Phys &P)
{
    double s[4] = {Ui[0], Ui[1], Ui[2], Ui[3]};
    squares<I>(s);
    double y[3] = {s[1], s[2], s[3]};
    Over(s[0]).all(y);
    const double d_temp = product<I>(P.c_temp, dv(Ui[4], Ui[0]) - xdiv::scale2<-1>(y[0] + y[1] + y[2]));
    const double sd = xi::root(d_temp);
    return product<I>(product<I>(product<I>(sd, sd), sd), dv(P.st1, d_temp + P.st));
}

// SSP-RK3 stage j and primitive recovery (Weno.cl:3084-3135).  Returns the
// new U in Un and writes FLOW fields rho,u,v,w,e,p,t,a into fo[9]
// (u,v,w,p,t,rho,mu,a,e order; mu untouched).
template <bool I>
__device__ __forceinline__ void rk_and_primitives(int j, double del_t, double mach, double det, const double U0[5],
                                                  const double U1[5], const double U2[5], const double L[5],
                                                  double Un[5], double &rho, double &u, double &v, double &w,
                                                  double &e, double &p, double &t, double &a_)
{
    const double l5[5] = {L[0], L[1], L[2], L[3], L[4]};
    if (j == 0) {
        double t[5];
        scaled<I>(del_t, l5, t);
#pragma unroll
        for (int c = 0; c < 5; ++c) Un[c] = U0[c] + t[c];
    } else if (j == 1) {
        const double z[5] = {U0[0], U0[1], U0[2], U0[3], U0[4]};
        double s[5], t[5];
        scaled<I>(3.0 / 4.0, z, s);
        scaled<I>(0.25 * del_t, l5, t);
#pragma unroll
        for (int c = 0; c < 5; ++c) Un[c] = s[c] + xdiv::scale2<-2>(U1[c]) + t[c];
    } else {
        double t[5], s[5], r[5], z[5] = {U0[0], U0[1], U0[2], U0[3], U0[4]};
        const double y[5] = {U2[0], U2[1], U2[2], U2[3], U2[4]};
        Over(3.0).all(z);
        scaled<I>(del_t, l5, t);
        scaled<I>(2.0 / 3.0, y, s);
        scaled<I>(2.0 / 3.0, t, r);
#pragma unroll
        for (int c = 0; c < 5; ++c) Un[c] = z[c] + s[c] + r[c];
    }
    double fu[5];
    {
        const double un[5] = {Un[0], Un[1], Un[2], Un[3], Un[4]};
        scaled<I>(dv(1.0, det), un, fu);
    }
    rho = fu[0];
    const Over d0(fu[0]);   // u, v, w, e, p / rho and 1.4 p / rho share the divisor
    double q[4] = {fu[1], fu[2], fu[3], fu[4]};
    d0.all(q);
    u = q[0];
    v = q[1];
    w = q[2];
    double s[3] = {u, v, w};
    squares<I>(s);
    e = q[3] - xdiv::scale2<-1>(s[0] + s[1] + s[2]);
    p = product<I>(product<I>(e, rho), 0.4);
    double r[2] = {p, product<I>(1.4, p)};
    d0.all(r);
    t = product<I>(1.4 * mach * mach, r[0]);
    a_ = xi::root(r[1]);
}

}  // namespace ex
}  // namespace cfd
