// lattice_fp64.cuh -- per-node operations of the FP64 lattice stage in the
// reference's evaluation order (physics_exact.cuh).  Include only from
// translation units compiled with --fmad=false.
//
// One RK stage j = prep (U_Q) -> visc (Viscous) -> face x3 + update (Weno).
// The update can also perform the next stage's prep on the values it just
// produced (fused form); the arithmetic is identical to a separate prep pass.
#pragma once

#include "lattice.cuh"
#include "physics_exact.cuh"

namespace cfd {
namespace ex {

// U_Q.cl for one node from primitives in registers: U_q = det*Q, Q, the
// contravariant node fluxes (Viscous.cl:560-631), sqrt(rho) and H.
template <bool I>
__device__ __forceinline__ void prep_values(const LatView &g, int n, int q, double rho, double u, double v, double w,
                                            double p)
{
    const int N = g.N;
    const double D = g.det[n];
    const double prim[5] = {rho, u, v, w, p};
    double Q[5], H;
    node_flux<I>(prim, [&](int c) { return g.m9[c * N + n]; }, D,
              [&](int d, int c, double f) { g.FEG[(d * 5 + c) * N + n] = f; }, Q, H);
#pragma unroll
    for (int c = 0; c < 5; ++c) g.Q[c * N + n] = Q[c];
    double *Uq = lat_U(g, q);
    {
        const double re[2] = {rho, Q[4]}, vel[3] = {u, v, w};
        double d[2], du[3];
        scaled<I>(D, re, d);
        scaled<I>(d[0], vel, du);
        Uq[0 * N + n] = d[0];
        Uq[1 * N + n] = du[0];
        Uq[2 * N + n] = du[1];
        Uq[3 * N + n] = du[2];
        Uq[4 * N + n] = d[1];
    }
    const double s = xi::root(rho), x[4] = {u, v, w, H};
    double sx[4];
    scaled<I>(s, x, sx);
    g.sh[n] = s;
#pragma unroll
    for (int c = 0; c < 4; ++c) g.sh[(1 + c) * N + n] = sx[c];
}

template <bool I = true>
__device__ __forceinline__ void prep_node(const LatView &g, int n, int q)
{
    const int N = g.N;
    prep_values<I>(g, n, q, g.prim9[LF_RHO * N + n], g.prim9[LF_U * N + n], g.prim9[LF_V * N + n],
                g.prim9[LF_W * N + n], g.prim9[LF_P * N + n]);
}

// The seven nodes at offsets -3..3 along d and their loc codes.
__device__ __forceinline__ void loc_line(const LatView &g, int i, int j, int k, int d, int s[7], int L[7])
{
#pragma unroll
    for (int o = 0; o < 7; ++o) {
        s[o] = lat_step(g, i, j, k, d, o - 3);
        L[o] = g.loc8[s[o]];
    }
}

// Viscous.cl on a lattice: derivatives of U_q (4th-order central on a
// periodic lattice, where every node has loc 0; the loc-code branches of
// Viscous.cl:285-332 on a lattice with loc codes; zero at ghosts, which no
// branch covers), viscous + MTS SGS fluxes, mu.
template <bool I>
__device__ __forceinline__ void visc_node(const LatView &g, int n, int q)
{
    const int N = g.N;
    const double *Uj = lat_U(g, q);
    int i, j, k;
    lat_ijk(g, n, i, j, k);
    double KS[3], Ui[5];
    const bool ghost = lat_ghost(g, n);
    // nodes outside the loc-code band take the central branch (the same
    // expression as the reference's central branch: the same bits)
    const unsigned lflag = g.locflag ? g.locflag[n] : 7u;
#pragma unroll
    for (int c = 0; c < 5; ++c) Ui[c] = Uj[c * N + n];
    auto dU = [&](int d, double (&out)[5]) {
        if (ghost) {
#pragma unroll
            for (int c = 0; c < 5; ++c) out[c] = 0.0;
        } else if (!lat_locdir(g, d) || !((lflag >> d) & 1u)) {
            const int at[5] = {lat_step(g, i, j, k, d, -2), lat_step(g, i, j, k, d, -1), n, lat_step(g, i, j, k, d, 1),
                               lat_step(g, i, j, k, d, 2)};
            central4<I>([&](int o, int c) { return Uj[c * N + at[o + 2]]; }, out);
        } else {
            int s[7], L[7];
            loc_line(g, i, j, k, d, s, L);
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                double f[7];
#pragma unroll
                for (int o = 0; o < 7; ++o) f[o] = Uj[c * N + s[o]];
                out[c] = visc_deriv_ref(f, L);
            }
        }
    };
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        const int m1 = lat_step(g, i, j, k, d, -1), p1 = lat_step(g, i, j, k, d, 1), c = d + 1;
        KS[d] = g.P.les && g.P.les != 2 ? ks_root(Uj[c * N + n], Ui[0], Uj[c * N + m1], Uj[m1], Uj[c * N + p1], Uj[p1]) : 0.0;
    }
    const double prim[5] = {g.prim9[LF_RHO * N + n], g.prim9[LF_U * N + n], g.prim9[LF_V * N + n],
                            g.prim9[LF_W * N + n], g.prim9[LF_P * N + n]};
    double mu;
    const double D = g.det[n];
    viscous_node<I>(dU, Ui, [&](int c) { return g.m9[c * N + n]; }, D, g.del ? g.del[n] : filter_width(D), prim, KS, g.P,
                 [&](int d, int c, double f) { g.V[(d * 5 + c) * N + n] = f; }, mu);
    g.prim9[LF_MU * N + n] = mu;
}

// Sutherland viscosity only (inviscid runs still report mu, Viscous.cl:458).
__device__ __forceinline__ void mu_node(const LatView &g, int n, int q)
{
    const int N = g.N;
    const double *Uj = lat_U(g, q);
    const double Ui[5] = {Uj[n], Uj[N + n], Uj[2 * N + n], Uj[3 * N + n], Uj[4 * N + n]};
    g.prim9[LF_MU * N + n] = mu_of<true>(Ui, g.P);
}

// Face n+1/2 along d (Weno.cl:336-3058 for that face, once) in four kernels
// (physics_exact.cuh), over the faces of a range of nodes: the Roe average and its scalars (base_node), one thread
// per characteristic field and correction component (char_node), one per
// component of the face states (back_node), two lanes per face for the LLF
// flux (flux_node).  What they hand on stays in a scratch of kFaceScratch
// doubles per face and direction.
enum { FS_BASE = 0, FS_POS = FB_N, FS_NEG = FS_POS + 5, FS_CA = FS_NEG + 5, FS_CB = FS_CA + 5, FS_QP = FS_CB + 5,
       FS_QN = FS_QP + 5, FS_KN = FS_QN + 5 };
static_assert(FS_KN == kFaceScratch && FS_KN + 3 == kFaceScratchNormals, "face scratch");

// The unit normal of a face, component c at [c * ld].
struct FaceNormal {
    const double *p;
    size_t ld;
    __device__ __forceinline__ double operator()(int c) const { return p[c * ld]; }
};

// The scratch column of node n, direction d: element s at [s * ld].  KN: the
// normals are in it.
template <bool KN>
__device__ __forceinline__ double *face_column(const FaceScratch &fs, int n, int d)
{
    return fs.p + (size_t)d * (KN ? kFaceScratchNormals : kFaceScratch) * fs.ld + (n - fs.n0);
}

template <bool KN>
__device__ __forceinline__ FaceNormal face_normal_at(const LatView &g, const FaceScratch &fs, const double *col, int n, int d)
{
    if (KN) return {col + (size_t)FS_KN * fs.ld, (size_t)fs.ld};
    return {g.kn + (size_t)d * 3 * g.N + n, (size_t)g.N};
}

__device__ __forceinline__ bool face_at(const LatView &g, int n, int d, int &i, int &j, int &k)
{
    lat_ijk(g, n, i, j, k);
    return lat_face_needed(g, i, j, k, d);
}

template <bool KN = false>
__device__ __forceinline__ void base_node(const LatView &g, const FaceScratch &fs, int n, int d)
{
    const int N = g.N;
    int i, j, k;
    if (!face_at(g, n, d, i, j, k)) return;
    const int rr = lat_step(g, i, j, k, d, 1);
    // sqrt(rho) and its products with u, v, w, H: left and right node
    const double sb = g.sh[rr], si = g.sh[n];
    double r[5], x[4];
    r[4] = sb * si;
#pragma unroll
    for (int c = 0; c < 4; ++c) x[c] = g.sh[(1 + c) * N + rr] + g.sh[(1 + c) * N + n];
    Over(sb + si).all(x);
#pragma unroll
    for (int c = 0; c < 4; ++c) r[c] = x[c];
    double B[FB_N], kn[3], *col = face_column<KN>(fs, n, d);
    if (KN) {
        face_normal(g.fm[(d * 3 + 0) * N + n], g.fm[(d * 3 + 1) * N + n], g.fm[(d * 3 + 2) * N + n], kn);
#pragma unroll
        for (int c = 0; c < 3; ++c) col[(size_t)(FS_KN + c) * fs.ld] = kn[c];
    } else {
        const FaceNormal k = face_normal_at<KN>(g, fs, col, n, d);
#pragma unroll
        for (int c = 0; c < 3; ++c) kn[c] = k(c);
    }
    face_base(r, kn, B);
#pragma unroll
    for (int s = 0; s < FB_N; ++s) col[(size_t)(FS_BASE + s) * fs.ld] = B[s];
}

// Every thread of the block calls it when Sync is the block's barrier; those
// past the range of nodes with active = false.
template <bool KN = false, class Sync = NoSync>
__device__ __forceinline__ void char_node(const LatView &g, const FaceScratch &fs, int n, int d, int q, bool active,
                                          const Sync &sync = Sync())
{
    const int N = g.N;
    int i, j, k;
    const bool face = active && face_at(g, n, d, i, j, k);
    double *col = face_column<KN>(fs, n, d);
    const FaceNormal kn = face_normal_at<KN>(g, fs, col, n, d);
    const size_t ld = fs.ld;
    int s[6];
    double pos, neg;
    char_pair(
        face,
        [&](double (&L)[5]) {
            left_row(q, [&](int e) { return col[(FS_BASE + e) * ld]; }, kn, L);
#pragma unroll
            for (int o = 0; o < 6; ++o) s[o] = lat_step(g, i, j, k, d, o - 2);
        },
        [&](int o, int c) { return g.Q[c * N + s[o]]; }, g.P.eps, pos, neg, sync);
    if (!face) return;
    col[(FS_POS + q) * ld] = pos;
    col[(FS_NEG + q) * ld] = neg;
}

template <bool KN = false>
__device__ __forceinline__ void back_node(const LatView &g, const FaceScratch &fs, int n, int d, int q)
{
    const int N = g.N;
    int i, j, k;
    if (!face_at(g, n, d, i, j, k)) return;
    double *col = face_column<KN>(fs, n, d);
    const size_t ld = fs.ld;
    double qp, qn;
    back_pair(q, [&](int s) { return col[(FS_BASE + s) * ld]; }, face_normal_at<KN>(g, fs, col, n, d),
              [&](int s) { return col[(FS_POS + s) * ld]; }, [&](int s) { return col[(FS_NEG + s) * ld]; }, qp, qn);
    col[(FS_QP + q) * ld] = qp;
    col[(FS_QN + q) * ld] = qn;
    const double *NF = g.FEG + (size_t)(d * 5 + q) * N;
    double f[6], ca, cb;
#pragma unroll
    for (int o = 0; o < 6; ++o) f[o] = NF[lat_step(g, i, j, k, d, o - 2)];
    correction_terms(f, ca, cb);
    col[(FS_CA + q) * ld] = ca;
    col[(FS_CB + q) * ld] = cb;
}

// lanes 2m and 2m + 1 of a warp: the pos and neg side of one face; lanes
// without a face take part with a face they do not store
template <bool KN = false>
__device__ __forceinline__ void flux_node(const LatView &g, const FaceScratch &fs, int n, int d, bool active)
{
    const int N = g.N;
    int i, j, k;
    const bool face = active && face_at(g, n, d, i, j, k);
    const int side = threadIdx.x & 1;
    const double *col = face_column<KN>(fs, n, d);
    const size_t ld = fs.ld;
    double q[5] = {1.0, 0.0, 0.0, 0.0, 2.5}, m[3] = {1.0, 0.0, 0.0}, det = 1.0, Fhat[5];
    if (face) {
#pragma unroll
        for (int c = 0; c < 5; ++c) q[c] = col[(FS_QP + 5 * side + c) * ld];
#pragma unroll
        for (int c = 0; c < 3; ++c) m[c] = g.fm[(d * 3 + c) * N + n];
        det = g.fdet[d * N + n];
    }
    llf_lanes(q, m[0], m[1], m[2], det, Fhat);
    if (!face) return;
#pragma unroll
    for (int c = 0; c < 5; ++c)   // components 0..2 on the even lane, 3..4 on the odd one
        if ((c >= 3) == (side != 0)) g.Fh[(d * 5 + c) * N + n] = Fhat[c] - col[(FS_CA + c) * ld] + col[(FS_CB + c) * ld];
}

// What the face and viscous kernels take from the geometry alone, once per
// solver: the unit normals of the faces along d (kn null: none) and the
// filter width.
__device__ __forceinline__ void geometry_node(const LatView &g, double *kn, double *del, int n, int d)
{
    const int N = g.N;
    if (d == 0) del[n] = filter_width(g.det[n]);
    if (!kn) return;
    double k[3];
    face_normal(g.fm[(d * 3 + 0) * N + n], g.fm[(d * 3 + 1) * N + n], g.fm[(d * 3 + 2) * N + n], k);
#pragma unroll
    for (int c = 0; c < 3; ++c) kn[(size_t)(d * 3 + c) * N + n] = k[c];
}

// Weno.cl:3060-3135 at one owned node (ghosts are the boundary routine's):
// L from the face fluxes and the viscous divergence (the loc-code branches
// of Weno.cl:2732-2856 on a lattice with loc codes), SSP-RK3 stage jst,
// primitives.  With fuse_next the node then runs the next stage's prep on
// the new primitives.
template <bool I>
__device__ __forceinline__ void update_node(const LatView &g, int n, int jst, bool fuse_next)
{
    const int N = g.N;
    if (lat_ghost(g, n)) {
        if (g.Lout) {
#pragma unroll
            for (int c = 0; c < 5; ++c) g.Lout[c * N + n] = 0.0;
        }
        return;
    }
    int i, j, k;
    lat_ijk(g, n, i, j, k);
    // the sum in the reference's order: the flux differences of the three
    // directions, then the viscous ones (loops: see viscous_node)
    double L[5];
    const unsigned lflag = g.locflag ? g.locflag[n] : 7u;   // as in visc_node
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        const int m1 = lat_step(g, i, j, k, d, -1);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const double df = g.Fh[(d * 5 + c) * N + n] - g.Fh[(d * 5 + c) * N + m1];
            L[c] = d == 0 ? df : L[c] + df;
        }
    }
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        double dvis[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        const double *Vd = g.V + (size_t)d * 5 * N;
        if (g.P.viscous && lat_locdir(g, d) && ((lflag >> d) & 1u)) {
            int s[7], B[7];
            loc_line(g, i, j, k, d, s, B);
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                double f[7];
#pragma unroll
                for (int o = 0; o < 7; ++o) f[o] = Vd[c * N + s[o]];
                dvis[c] = weno_visc_deriv_ref(f, B);
            }
        } else if (g.P.viscous) {
            const int at[5] = {lat_step(g, i, j, k, d, -2), lat_step(g, i, j, k, d, -1), n, lat_step(g, i, j, k, d, 1),
                               lat_step(g, i, j, k, d, 2)};
            central4<I>([&](int o, int c) { return Vd[c * N + at[o + 2]]; }, dvis);
        }
#pragma unroll
        for (int c = 0; c < 5; ++c) L[c] = L[c] + dvis[c];
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) L[c] = (-1.0) * L[c];
    if (g.Lout) {
#pragma unroll
        for (int c = 0; c < 5; ++c) g.Lout[c * N + n] = L[c];
    }
    double u0[5], u1[5], u2[5], Un[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) { u0[c] = g.U0[c * N + n]; u1[c] = g.U1[c * N + n]; u2[c] = g.U2[c * N + n]; }
    double rho, u, v, w, e, p, t, a;
    rk_and_primitives<I>(jst, g.dt, g.P.mach, g.det[n], u0, u1, u2, L, Un, rho, u, v, w, e, p, t, a);
    double *Uo = jst == 0 ? g.U1 : (jst == 1 ? g.U2 : g.U0);
#pragma unroll
    for (int c = 0; c < 5; ++c) Uo[c * N + n] = Un[c];
    g.prim9[LF_RHO * N + n] = rho;
    g.prim9[LF_U * N + n] = u;
    g.prim9[LF_V * N + n] = v;
    g.prim9[LF_W * N + n] = w;
    g.prim9[LF_E * N + n] = e;
    g.prim9[LF_P * N + n] = p;
    g.prim9[LF_T * N + n] = t;
    g.prim9[LF_A * N + n] = a;
    if (!(isfinite(rho) && isfinite(u) && isfinite(v) && isfinite(w) && isfinite(p))) atomicOr(g.flags, 2u);
    if (fuse_next) prep_values<I>(g, n, jst == 2 ? 0 : jst + 1, rho, u, v, w, p);
}

}  // namespace ex
}  // namespace cfd
