// physics.cuh -- device arithmetic of the RHS path, shared by the drop-in
// (reference-layout) kernels and the structured face-based kernels.
//
// Every function follows the reference kernels' formulas (cited per
// function) with gamma = 1.4 written as the reference writes it (0.4, 1.4,
// 0.2).  Functions are templated on the compute type T; the mixed-precision
// form instantiates them with float (the FP64 form uses the exact-order
// restatement in physics_exact.cuh).  Repeated divisors are inverted once.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace cfd {

// Quotient, square root and its reciprocal.  The float forms are the
// hardware approximations (about 2 ulp) with subnormal operands and results
// taken as zero: the forms that keep subnormals scale their operand into
// range and the result back, four instructions more at each of a face's 54
// (physics_x2.cuh; a face direction of the split TGV 128^3 0.118 -> 0.107 ms).  Their operands here are
// densities, sums with the WENO epsilon, sound speeds and metrics, none
// within 2^-60 of that range.  Other types compute exactly.
__device__ __forceinline__ float frcp(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float fsqrt(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float frsqrt(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
template <class T> __device__ __forceinline__ T qdiv(T a, T b) { return a / b; }
template <> __device__ __forceinline__ float qdiv<float>(float a, float b) { return a * frcp(b); }
template <class T> __device__ __forceinline__ T qsqrt(T x) { return sqrt(x); }
template <> __device__ __forceinline__ float qsqrt<float>(float x) { return fsqrt(x); }

// Sums of products with their contraction written out, so that every kernel
// that evaluates a face (tiles of any shape, the batched stage) rounds it
// alike: a b + c d, a b - c d, a b + c d + e f.
__device__ __forceinline__ float dot2(float a, float b, float c, float d) { return fmaf(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ float det2(float a, float b, float c, float d) { return fmaf(a, b, -__fmul_rn(c, d)); }
__device__ __forceinline__ float dot3(float a, float b, float c, float d, float e, float f)
{
    return fmaf(a, b, dot2(c, d, e, f));
}

// Roe-averaged face state from the two adjacent nodes (U_Q.cl:60-109):
// out = {u, v, w, h, rho}.  sb/hb belong to the neighbour, si/hi to the node.
__device__ __forceinline__ void roe_average(float sb, float ub, float vb, float wb, float hb, float si, float ui,
                                            float vi, float wi, float hi, float out[5])
{
    const float iden = frcp(sb + si);
    out[4] = __fmul_rn(sb, si);
    out[0] = __fmul_rn(dot2(sb, ub, si, ui), iden);
    out[1] = __fmul_rn(dot2(sb, vb, si, vi), iden);
    out[2] = __fmul_rn(dot2(sb, wb, si, wi), iden);
    out[3] = __fmul_rn(dot2(sb, hb, si, hi), iden);
}

// Roe eigen-system of one face (Weno.cl:337-413): k_bar = grad(zeta)/|grad(zeta)|
// from the face metric, sound speed from the Roe state, and what the left and
// right eigenvectors of the Euler flux Jacobian along k_bar are made of
// (physics_x2.cuh left_times, right_times2).
struct FaceEigen {
    float kx, ky, kz, ru, rv, rw, h2, g2;             // unit normal; Roe velocities, |u|^2/2; 0.4 / a^2
    float ix, iy, iz, b4, ba, nx, ny, nz, al, ala, ae;

    __device__ __forceinline__ void init(float mx, float my, float mz, const float roe[5])
    {
        ru = roe[0];
        rv = roe[1];
        rw = roe[2];
        const float rh = roe[3], rr = roe[4];
        const float ikk = frsqrt(dot3(mx, mx, my, my, mz, mz));
        kx = __fmul_rn(mx, ikk);
        ky = __fmul_rn(my, ikk);
        kz = __fmul_rn(mz, ikk);
        h2 = __fmul_rn(0.5f, dot3(ru, ru, rv, rv, rw, rw));
        const float a2 = __fmul_rn(0.4f, __fsub_rn(rh, h2)), a = fsqrt(a2), ia = frcp(a), irr = frcp(rr);
        constexpr float is2 = 0.70710678118654752f;   // 1 / sqrt(2)
        const float rs = __fmul_rn(rr, is2), irs = __fmul_rn(irr, is2);
        g2 = __fmul_rn(0.4f, __fmul_rn(ia, ia));
        ix = __fmul_rn(kx, irr);
        iy = __fmul_rn(ky, irr);
        iz = __fmul_rn(kz, irr);
        nx = __fmul_rn(kx, rr);
        ny = __fmul_rn(ky, rr);
        nz = __fmul_rn(kz, rr);
        al = __fmul_rn(rs, ia);              // alpha = rho / (sqrt(2) a)
        ala = rs;                            // alpha a
        ae = __fmul_rn(__fmul_rn(rs, a), 2.5f);   // alpha a^2 / 0.4
        b4 = __fmul_rn(__fmul_rn(irs, ia), 0.4f); // 0.4 / (sqrt(2) rho a)
        ba = irs;                            // beta a
    }
};

// Branch selection of the location-code-driven first derivative of the
// Viscous kernel (Viscous.cl:285-332; the same set for eta and xi) from the
// loc codes L[0..6] of offsets -3..3.  The reference tests its branches in
// sequence and the last match wins: 1 one-sided backward, 2 one-sided
// forward, 3/4 biased next to a boundary node, 5 central; 0 = no branch
// (the derivative is 0).
__host__ __device__ __forceinline__ int visc_branch(const int L[7])
{
    const int L0 = L[3];
    int b = 0;
    if (L0 > 0 && L0 <= 52 && L[4] == 100) b = 1;
    if (L0 > 0 && L0 <= 52 && L[2] == 100) b = 2;
    if (L0 == 0 && L[4] > 0 && L[4] <= 52 && L[5] == 100) b = 3;
    if (L0 == 0 && L[2] > 0 && L[1] == 100) b = 4;
    if (L0 == 0 && L[1] != 100 && L[2] != 100 && L[5] != 100 && L[4] != 100) b = 5;
    if (L0 > 0 && L[1] != 100 && L[2] != 100 && L[5] != 100 && L[4] != 100) b = 5;
    return b;
}

// Viscous-flux derivative branches of the Weno kernel (Weno.cl:2732-2856):
// central unless a one-sided or biased branch matches.  The reference has
// no branch for a boundary node away from ghosts in a direction (its value
// is uninitialised there); the central form is used.
__host__ __device__ __forceinline__ int weno_visc_branch(const int L[7])
{
    const int L0 = L[3];
    int b = 5;
    if (L0 > 0 && L0 <= 52 && L[4] == 100) b = 1;
    if (L0 > 0 && L0 <= 52 && L[2] == 100) b = 2;
    if (L0 == 0 && L[4] > 0 && L[4] <= 52 && L[5] == 100) b = 3;
    if (L0 == 0 && L[2] > 0 && L[2] <= 52 && L[1] == 100) b = 4;
    return b;
}

// The derivative of branch b from the values f[0..6] at offsets -3..3, as
// the reference writes each formula.
template <class T>
__device__ __forceinline__ T branch_deriv(int b, const T f[7])
{
    switch (b) {
    case 1: return (T(1.0) / T(6.0)) * (T(11.0) * f[3] - T(18.0) * f[2] + T(9.0) * f[1] - T(2.0) * f[0]);
    case 2: return (T(1.0) / T(6.0)) * (T(-11.0) * f[3] + T(18.0) * f[4] - T(9.0) * f[5] + T(2.0) * f[6]);
    case 3: return (T(1.0) / T(6.0)) * (T(2.0) * f[4] + T(3.0) * f[3] - T(6.0) * f[2] + f[1]);
    case 4: return (T(1.0) / T(6.0)) * ((T(-2.0)) * f[2] - T(3.0) * f[3] + T(6.0) * f[4] - f[5]);
    case 5: return (T(1.0) / T(12.0)) * (T(8.0) * (f[4] - f[2]) - (f[5] - f[1]));
    default: return T(0.0);
    }
}

__device__ __forceinline__ double visc_deriv_ref(const double f[7], const int L[7])
{
    return branch_deriv<double>(visc_branch(L), f);
}

__device__ __forceinline__ double weno_visc_deriv_ref(const double f[7], const int L[7])
{
    return branch_deriv<double>(weno_visc_branch(L), f);
}

// Physical constants of one run.
struct Phys {
    double mach, reynolds, prandtl, t_inf, eps;
    int viscous, les;   // les: 0 none, 1 mixed time scale, 2 Smagorinsky
    double cs;          // Smagorinsky C_s
    // constants of the viscous terms, in the reference's own operations
    // (make_phys): 1.4 M^2 0.4, 110.4 / T_inf, 1 + that, Pr Re, 1 / (0.56 M^2)
    double c_temp, st, st1, pr_re, ck;
};

// Viscous and SGS fluxes at one node from the derivatives of U along the
// three directions (Viscous.cl:439-631) in FP32, contraction written out
// (as for the face).  dU[d][c]: derivative of U_c along direction d; Ui: U
// at the node; m: node metrics (9); det: node det; DEL: the filter width
// det^(-1/3); prim: rho,u,v,w,p of FLOW at the node; KS: the magnitudes of
// the three MTS test-filter velocity differences (the roots of the
// reference's KS).  Writes contravariant Fv/Ev/Gv (x det) and mu.
__device__ __forceinline__ void viscous_node_flux(const float dU[3][5], const float Ui[5], const float m[9], float det,
                                                  float DEL, const float prim[5], const float KS[3], const Phys &P,
                                                  float Fv[5], float Ev[5], float Gv[5], float &mu_out)
{
    auto mul = [](float a, float b) { return __fmul_rn(a, b); };
    const float Mach = (float)P.mach, Reyl = (float)P.reynolds, Pr = (float)P.prandtl, Free_t = (float)P.t_inf;
    const float iU0 = frcp(Ui[0]);
    const float uu = mul(Ui[1], iU0), vv = mul(Ui[2], iU0), ww = mul(Ui[3], iU0), ee = mul(Ui[4], iU0);
    float uc[3], vc[3], wc[3], tc[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        uc[d] = mul(iU0, fmaf(-uu, dU[d][0], dU[d][1]));
        vc[d] = mul(iU0, fmaf(-vv, dU[d][0], dU[d][2]));
        wc[d] = mul(iU0, fmaf(-ww, dU[d][0], dU[d][3]));
        tc[d] = fmaf(iU0, fmaf(-ee, dU[d][0], dU[d][4]), -dot3(uu, uc[d], vv, vc[d], ww, wc[d]));
    }
    // Sutherland's law with T = gamma M^2 (gamma-1) e (Viscous.cl:451-458)
    const float d_temp = mul(1.4f * 0.4f * Mach * Mach, fmaf(-0.5f, dot3(uu, uu, vv, vv, ww, ww), ee));
    const float sd = fsqrt(d_temp);
    const float S = qdiv(110.4f, Free_t);
    const float mu = mul(mul(mul(sd, sd), sd), qdiv(1.0f + S, d_temp + S));
    mu_out = mu;
    float gu[3], gv[3], gw[3], gt[3];   // gradients along x, y, z
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        gu[x] = dot3(uc[0], m[x], uc[1], m[3 + x], uc[2], m[6 + x]);
        gv[x] = dot3(vc[0], m[x], vc[1], m[3 + x], vc[2], m[6 + x]);
        gw[x] = dot3(wc[0], m[x], wc[1], m[3 + x], wc[2], m[6 + x]);
        gt[x] = dot3(tc[0], m[x], tc[1], m[3 + x], tc[2], m[6 + x]);
    }
    const float sxy = gu[1] + gv[0], sxz = gu[2] + gw[0], syz = gv[2] + gw[1];
    const float kq = -mul(mul(mu, 1.4f), qdiv(1.0f, Pr * Reyl));   // Viscous.cl:461-463
    const float mr = mul(mu, qdiv(1.0f, Reyl));                    // Viscous.cl:466-476
    const float trace = mul(-2.0f / 3.0f, gu[0] + gv[1] + gw[2]);
    // stress and heat flux, the molecular part; the SGS part is added below
    float txx = -mul(mr, fmaf(2.0f, gu[0], trace)), tyy = -mul(mr, fmaf(2.0f, gv[1], trace)),
          tzz = -mul(mr, fmaf(2.0f, gw[2], trace));
    float txy = -mul(mr, sxy), txz = -mul(mr, sxz), tyz = -mul(mr, syz);
    const float u = prim[1], v = prim[2], w = prim[3];
    float ex = fmaf(kq, gt[0], dot3(u, txx, v, txy, w, txz)), ey = fmaf(kq, gt[1], dot3(u, txy, v, tyy, w, tyz)),
          ez = fmaf(kq, gt[2], dot3(u, txz, v, tyz, w, tzz));
    if (P.les) {  // SGS model: mixed time scale (Viscous.cl:490-558) or Smagorinsky
        const float C_MTS = 0.03f, iC_T = 0.1f;
        const float off = mul(0.25f, dot3(sxy, sxy, syz, syz, sxz, sxz));   // sum of (s_ij / 2)^2
        const float dia = dot3(gu[0], gu[0], gv[1], gv[1], gw[2], gw[2]);
        float ed[3];
        if (P.les == 2) {   // (C_s Delta)^2 |S|, |S| = sqrt(2 S_ij S_ij), Delta = det^(1/3) = 1/DEL
            const float ls = qdiv((float)P.cs, DEL);
            ed[0] = ed[1] = ed[2] = mul(mul(ls, ls), fsqrt(dot2(2.0f, dia, 4.0f, off)));
        } else {
            const float mod = fsqrt(mul(2.0f, fmaf(2.0f / 3.0f, dia, off)));
            const float dm = mul(DEL, mod), cd = mul(C_MTS, DEL);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const float sk = KS[d];
                const float e0 = mul(cd, sk);
                ed[d] = mod != 0.0f ? mul(frcp(fmaf(qdiv(dm, sk), iC_T, 1.0f)), e0) : e0;
            }
        }
        const float r2 = mul(-2.0f, Ui[0]);
        const float r0 = mul(r2, ed[0]), r1 = mul(r2, ed[1]), rz = mul(r2, ed[2]);
        const float TXY = mul(r0, mul(0.5f, sxy)), TYZ = mul(r1, mul(0.5f, syz)), TXZ = mul(rz, mul(0.5f, sxz));
        const float TXX = mul(r0, gu[0]), TYY = mul(r1, gv[1]), TZZ = mul(rz, gw[2]);
        const float kQ = mul(-1.4f, qdiv(1.0f, 1.4f * 0.4f * Mach * Mach));   // Q and its 0.4 Q share
        ex += fmaf(mul(kQ, ed[0]), gt[0], mul(TXX + TXY + TXZ, u));
        ey += fmaf(mul(kQ, ed[1]), gt[1], mul(TXY + TYY + TYZ, v));
        ez += fmaf(mul(kQ, ed[2]), gt[2], mul(TXZ + TYZ + TZZ, w));
        txx += TXX;
        tyy += TYY;
        tzz += TZZ;
        txy += TXY;
        txz += TXZ;
        tyz += TYZ;
    }
    // Cartesian viscous fluxes, Viscous.cl:580-596, through the metrics
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float *o = d == 0 ? Fv : (d == 1 ? Ev : Gv);
        const float mx = mul(det, m[3 * d]), my = mul(det, m[3 * d + 1]), mz = mul(det, m[3 * d + 2]);
        o[0] = 0.0f;
        o[1] = dot3(mx, txx, my, txy, mz, txz);
        o[2] = dot3(mx, txy, my, tyy, mz, tyz);
        o[3] = dot3(mx, txz, my, tyz, mz, tzz);
        o[4] = dot3(mx, ex, my, ey, mz, ez);
    }
}

// Contravariant node inviscid flux along one direction (x det) from the
// primitives, Viscous.cl:560-578 and 615-631, in FP32:
// det (m . U) q + p det m.
__device__ __forceinline__ void node_inviscid_flux(const float prim[5], const float m[3], float det, float o[5])
{
    const float rho = prim[0], u = prim[1], v = prim[2], w = prim[3], p = prim[4];
    const float ke = __fmul_rn(__fmul_rn(0.5f, rho), dot3(u, u, v, v, w, w));
    const float Et = fmaf(p, 3.5f, ke);
    const float mx = __fmul_rn(det, m[0]), my = __fmul_rn(det, m[1]), mz = __fmul_rn(det, m[2]);
    const float un = dot3(mx, u, my, v, mz, w), ru = __fmul_rn(rho, un);
    o[0] = ru;
    o[1] = dot2(ru, u, mx, p);
    o[2] = dot2(ru, v, my, p);
    o[3] = dot2(ru, w, mz, p);
    o[4] = __fmul_rn(Et, un);
}

}  // namespace cfd
