// dropin.cu -- the three reference kernels on the reference's own layout.
//
// One thread per row (work-item), exactly the NDRange of the reference
// (Solver.cpp:31-38, local size 1 there).  Buffers are the packed AoS structs
// of include/cfd_rhs.h; device code reads them through aligned double/int
// views (every struct size is a multiple of 8 bytes) rather than through the
// packed types, which would force byte-wise loads.  Neighbour chains are
// bounds-checked: a row whose stencil leaves [0, n_rows) is skipped and the
// context's error word gets CFD_FLAG_BAD_INDEX.
//
// Arithmetic: the exact FP64 layer (physics_exact.cuh); this file is
// compiled with --fmad=false so that results follow the reference's
// evaluation order.
//
// Weno evaluates both faces of each direction at every row, so every
// interior face is computed twice from identical inputs (as row n's +1/2
// face and as row n+1's -1/2 face).  With a scratch buffer the launch is
// split: the k_row_* kernels compute each row's +1/2 face once and, where
// its plus neighbour p has this row as its minus neighbour and every input
// of p's -1/2 face is bit-identical (then so are the stencil rows; face
// metric, face det and Roe state are compared), also store it as p's -1/2
// face, stamped with the call's generation; k_weno_minus computes the -1/2
// faces left unstamped (box edges, loc codes, inconsistent tables), and
// k_weno<true> reads both faces from the scratch.  The results are the same
// bits either way.
//
// The k_row_* kernels are the lattice face pass (faces_fp64.cu: the FP64
// pipe runs the sums, the integer pipe the products, quotients and roots,
// so many small threads) on rows: one thread per face, characteristic
// field, component and side, in rounds of kRowRound rows.  The first also
// notes the six stencil rows, so that the neighbour chain (five loads that
// wait for one another) is walked once per face instead of ten times.  TGV
// 96^3: cfd_weno 8.9 -> 4.8 ms.
#include <algorithm>

#include "internal.h"
#include "physics_exact.cuh"

namespace cfd {

// ---- aligned views of the packed reference structs ----
// GRID: 56 B = 7 doubles = 14 ints; x,y,z at doubles 0..2, N0..N5 at ints
// 6..11, ID at 12, loc at 13.
__device__ __forceinline__ int grid_nb(const int *g, int row, int which) { return g[14 * row + 6 + which]; }
__device__ __forceinline__ int grid_loc(const int *g, int row) { return g[14 * row + 13]; }
// neighbour slot of (+d) and (-d): d=0 -> N1/N3, d=1 -> N0/N2, d=2 -> N4/N5
__device__ __forceinline__ int plus_slot(int d) { return d == 0 ? 1 : (d == 1 ? 0 : 4); }
__device__ __forceinline__ int minus_slot(int d) { return d == 0 ? 3 : (d == 1 ? 2 : 5); }

// Chained neighbour gather (Weno.cl:159-226): idx[d][o+3], o = -3..3.
// Returns false if any index leaves [0, n_rows).
__device__ __forceinline__ bool gather_star(const int *grid, int gid, int n_rows, int idx[3][7])
{
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        idx[d][3] = gid;
        int p = gid, m = gid;
#pragma unroll
        for (int o = 1; o <= 3; ++o) {
            p = grid_nb(grid, p, plus_slot(d));
            m = grid_nb(grid, m, minus_slot(d));
            if ((unsigned)p >= (unsigned)n_rows || (unsigned)m >= (unsigned)n_rows) return false;
            idx[d][3 + o] = p;
            idx[d][3 - o] = m;
        }
    }
    return true;
}

// The seven rows of direction d of a star that gather_star has checked.
__device__ __forceinline__ void star_line(const int *grid, int gid, int d, int s[7])
{
    s[3] = gid;
#pragma unroll
    for (int o = 1; o <= 3; ++o) {
        s[3 + o] = grid_nb(grid, s[2 + o], plus_slot(d));
        s[3 - o] = grid_nb(grid, s[4 - o], minus_slot(d));
    }
}

// The derivative of branch b (physics.cuh) from seven rows of one component
// (stride 5), out of line: rows next to ghosts take it, the others the
// central form.
static __device__ __noinline__ double row_deriv(const double *x, int i0, int i1, int i2, int i3, int i4, int i5, int i6,
                                                int b)
{
    const double f[7] = {x[5 * (size_t)i0], x[5 * (size_t)i1], x[5 * (size_t)i2], x[5 * (size_t)i3],
                         x[5 * (size_t)i4], x[5 * (size_t)i5], x[5 * (size_t)i6]};
    return branch_deriv<double>(b, f);
}

// FLOW field offsets inside the 9-double row
enum { FU = 0, FV = 1, FW = 2, FP = 3, FT = 4, FRHO = 5, FMU = 6, FA = 7, FE = 8 };

// ------------------------------------------------------------------ U_Q --
// sqrt(rho) of every row and its products with u, v, w and the total
// enthalpy (U_Q.cl:60-65), once per row: sh[5*row ..].  k_uq<true> reads
// them for the row and its six neighbours instead of evaluating them seven
// times.
__global__ void __launch_bounds__(128) k_uq_node(const double *__restrict__ flow, int n_rows, double *__restrict__ sh)
{
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n_rows) return;
    const double *f = flow + 9 * (size_t)row;
    const double rho = f[FRHO], u = f[FU], v = f[FV], w = f[FW];
    const double s = xi::root(rho), x[4] = {u, v, w, ex::enthalpy(rho, u, v, w, f[FP])};
    double sx[4];
    ex::scaled<true>(s, x, sx);
    double *o = sh + 5 * (size_t)row;
    o[0] = s;
#pragma unroll
    for (int c = 0; c < 4; ++c) o[1 + c] = sx[c];
}

// U_Q.cl:36-125.
template <bool SH>
__global__ void __launch_bounds__(128) k_uq(double *__restrict__ U, double *__restrict__ Q,
                                            const int *__restrict__ grid, const double *__restrict__ det,
                                            const double *__restrict__ flow, double *__restrict__ roe, int n_items,
                                            int n_rows, unsigned *flags, const double *__restrict__ sh)
{
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n_items) return;
    int nb[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        nb[s] = grid_nb(grid, gid, s);
        if ((unsigned)nb[s] >= (unsigned)n_rows) {
            atomicOr(flags, CFD_FLAG_BAD_INDEX);
            return;
        }
    }
    const double *fi = flow + 9 * (size_t)gid;
    const double rho = fi[FRHO], u = fi[FU], v = fi[FV], w = fi[FW], p = fi[FP];
    const double si = SH ? sh[5 * (size_t)gid] : sqrt(rho);
    const double hi = SH ? 0.0 : ex::enthalpy(rho, u, v, w, p);
    // ROE block order ip, jp, kp, im, jm, km: block d is the +d face
    // (neighbour slot plus_slot(d)), block d + 3 the -d face (minus_slot(d)).
    //
    // With SH the Roe state of a face is evaluated once.  roe() is symmetric
    // in its two rows bit for bit (one product, and a sum of two products
    // over a sum: IEEE addition and multiplication commute), so the +d
    // block of row m equals the -d block of row q = plus(m) whenever
    // minus(q) == m.  Row m then also stores it as q's -d block, provided q
    // is a row of this launch, and row q skips that block: both rows test
    // the same predicate (m, q < n_items, plus(m) == q, minus(q) == m), so
    // every block has exactly one writer.
    double *r = roe + 36 * (size_t)gid;
#pragma unroll
    for (int b = 0; b < 6; ++b) {
        const int d = b % 3;
        const bool plus = b < 3;
        const int nr = nb[plus ? plus_slot(d) : minus_slot(d)];
        if (SH && !plus && nr < n_items && grid_nb(grid, nr, plus_slot(d)) == gid) continue;
        double ra[5];
        if (SH) {   // the same sums of products over the same sum
            const double *sn = sh + 5 * (size_t)nr, *sg = sh + 5 * (size_t)gid;
            const double sb = sn[0];
            double x[4] = {sn[1] + sg[1], sn[2] + sg[2], sn[3] + sg[3], sn[4] + sg[4]};
            ex::Over(sb + si).all(x);
#pragma unroll
            for (int c = 0; c < 4; ++c) ra[c] = x[c];
            ra[4] = xi::mul(sb, si);
        } else {
            const double *fn = flow + 9 * (size_t)nr;
            const double rb = fn[FRHO], ub = fn[FU], vb = fn[FV], wb = fn[FW];
            ex::roe(sqrt(rb), ub, vb, wb, ex::enthalpy(rb, ub, vb, wb, fn[FP]), si, u, v, w, hi, ra);
        }
        r[6 * b + 0] = ra[0];
        r[6 * b + 1] = ra[1];
        r[6 * b + 2] = ra[2];
        r[6 * b + 4] = ra[3];
        r[6 * b + 5] = ra[4];
        if (SH && plus && nr < n_items && grid_nb(grid, nr, minus_slot(d)) == gid) {
            double *rq = roe + 36 * (size_t)nr + 6 * (d + 3);
            rq[0] = ra[0];
            rq[1] = ra[1];
            rq[2] = ra[2];
            rq[4] = ra[3];
            rq[5] = ra[4];
        }
    }
    const double D = det[gid];
    double s[3] = {u, v, w}, q[3], du[3], d2[2];
    const double vel[3] = {u, v, w};
    xi::sq_n(s);
    const double E = ex::dv(p, 0.4) + xi::mul(xdiv::scale2<-1>(rho), s[0] + s[1] + s[2]);   // 0.5 rho: same bits
    const double re[2] = {rho, E};
    ex::scaled<true>(rho, vel, q);
    ex::scaled<true>(D, re, d2);
    ex::scaled<true>(d2[0], vel, du);
    double *Ur = U + 5 * (size_t)gid, *Qr = Q + 5 * (size_t)gid;
    Ur[0] = d2[0];
    Ur[1] = du[0];
    Ur[2] = du[1];
    Ur[3] = du[2];
    Ur[4] = d2[1];
    Qr[0] = rho;
    Qr[1] = q[0];
    Qr[2] = q[1];
    Qr[3] = q[2];
    Qr[4] = E;
}

// -------------------------------------------------------------- Viscous --
// Viscous.cl:23-643.
// The inviscid node fluxes and the filter width of every row (their own
// kernel: beside the viscous fluxes they would spill; in one: TGV 96^3 1.17 ms
// at 3 blocks per SM, 1.38 at 4, with 3 KB of spill loads per thread) but
// those k_viscous skips.  The width waits in component 0 of the row's own Fv,
// which k_viscous writes after reading it: no memory but the call's outputs,
// so calls on different streams share nothing.
template <bool I>
__global__ void __launch_bounds__(128, 6) k_node_flux(double *__restrict__ F, double *__restrict__ E,
                                                      double *__restrict__ G, double *__restrict__ Fv,
                                                      const int *__restrict__ grid, const double *__restrict__ metric,
                                                      const double *__restrict__ det, const double *__restrict__ flow,
                                                      int n_items, int n_rows, int les)
{
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n_items) return;
    {
        int idx[3][7];
        if (!gather_star(grid, gid, n_rows, idx)) return;
    }
    const double D = det[gid];
    const double *m = metric + 63 * (size_t)gid;
    const double *fr = flow + 9 * (size_t)gid;
    const double prim[5] = {fr[FRHO], fr[FU], fr[FV], fr[FW], fr[FP]};
    double Qn[5], H;
    ex::node_flux<I>(prim, [&](int k) { return m[k]; }, D,
                  [&](int e, int c, double f) { (e == 0 ? F : (e == 1 ? E : G))[5 * (size_t)gid + c] = f; }, Qn, H);
    if (les) Fv[5 * (size_t)gid] = ex::filter_width(D);
}

// After k_node_flux.  TGV 96^3, both kernels: 1.00 ms at 3 or 4 blocks of 128
// per SM, 1.19 at 5.  The integer form in blocks of 256, which share its long
// code better: 0.73 -> 0.69 ms for both kernels (0.72 with the check of the
// neighbour chain in both).
template <bool I>
constexpr int kViscousThreads = I ? 256 : 128;
template <bool I>
__global__ void __launch_bounds__(kViscousThreads<I>, 512 / kViscousThreads<I>)
k_viscous(Phys P, const double *__restrict__ U, double *__restrict__ Fv, double *__restrict__ Ev,
          double *__restrict__ Gv, const int *__restrict__ grid, const double *__restrict__ metric,
          const double *__restrict__ det, double *__restrict__ flow, int n_items, int n_rows, unsigned *flags)
{
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n_items) return;
    {
        int idx[3][7];
        if (!gather_star(grid, gid, n_rows, idx)) {
            atomicOr(flags, CFD_FLAG_BAD_INDEX);
            return;
        }
    }
    const double *m = metric + 63 * (size_t)gid;
    const double D = det[gid];
    const double *fr = flow + 9 * (size_t)gid;
    const double prim[5] = {fr[FRHO], fr[FU], fr[FV], fr[FW], fr[FP]};
    auto metric_at = [&](int k) { return m[k]; };
    double mu;
    {
        // the star is walked again for each direction (it is cached by now):
        // its 18 rows would not fit the registers beside the fluxes
        auto dU = [&](int d, double (&out)[5]) {
            int s[7], L[7];
            star_line(grid, gid, d, s);
#pragma unroll
            for (int o = 0; o < 7; ++o) L[o] = grid_loc(grid, s[o]);
            const int b = visc_branch(L);
            if (b == 5) {
                ex::central4<I>([&](int o, int c) { return U[5 * (size_t)s[o + 3] + c]; }, out);
                return;
            }
#pragma unroll
            for (int c = 0; c < 5; ++c) out[c] = row_deriv(U + c, s[0], s[1], s[2], s[3], s[4], s[5], s[6], b);
        };
        double Ui[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) Ui[c] = U[5 * (size_t)gid + c];
        double KS[3];   // MTS test filter (Viscous.cl:493-495)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int c = d + 1;
            const double *um = U + 5 * (size_t)grid_nb(grid, gid, minus_slot(d)),
                         *up = U + 5 * (size_t)grid_nb(grid, gid, plus_slot(d));
            KS[d] = P.les && P.les != 2 ? ex::ks_root(Ui[c], Ui[0], um[c], um[0], up[c], up[0]) : 0.0;
        }
        ex::viscous_node<I>(dU, Ui, metric_at, D, P.les ? Fv[5 * (size_t)gid] : 0.0, prim, KS, P,
                         [&](int e, int c, double f) {
                             (e == 0 ? Fv : (e == 1 ? Ev : Gv))[5 * (size_t)gid + c] = P.viscous ? f : 0.0;
                         },
                         mu);
    }
    flow[9 * (size_t)gid + FMU] = mu;
}

// ----------------------------------------------------------------- Weno --
// Corrected face flux of row gid, direction d, side s (0: +1/2, 1: -1/2)
// from the row's own face data (metric block 1+2d+s, DETERM 2d+s, ROE
// block d+3s) over the stencil rows st[0..5] (offsets -2..3 for s = 0,
// -3..2 for s = 1), Weno.cl:336-3058.
__device__ __forceinline__ void face_side(const Phys &P, int gid, int d, int s, const int st[6],
                                          const double *__restrict__ deter, const double *__restrict__ Q,
                                          const double *__restrict__ metric, const double *__restrict__ roe,
                                          const double *__restrict__ NF, double Fh[5])
{
    const double *fm = metric + 63 * (size_t)gid + 9 * (1 + 2 * d + s) + 3 * d;
    const double det_f = deter[6 * (size_t)gid + 2 * d + s];
    const double *ra = roe + 36 * (size_t)gid + 6 * (d + 3 * s);
    const double rstate[5] = {ra[0], ra[1], ra[2], ra[4], ra[5]};
    double pts[6][5], nfv[6];
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int c = 0; c < 5; ++c) pts[k][c] = Q[5 * (size_t)st[k] + c];
    double Fhat[5];
    ex::face_flux(pts, fm[0], fm[1], fm[2], det_f, rstate, P.eps, Fhat);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
#pragma unroll
        for (int k = 0; k < 6; ++k) nfv[k] = NF[5 * (size_t)st[k] + c];
        Fh[c] = ex::corrected(Fhat[c], nfv);
    }
}

// Rows of offsets -2..3 of row n along d (chained neighbours); false if the
// chain leaves [0, n_rows).
__device__ __forceinline__ bool plus_line(const int *grid, int n, int n_rows, int d, int st[6])
{
    st[2] = n;
    int m = n, p = n;
#pragma unroll
    for (int o = 1; o <= 3; ++o) {
        p = grid_nb(grid, p, plus_slot(d));
        if ((unsigned)p >= (unsigned)n_rows) return false;
        st[2 + o] = p;
        if (o <= 2) {
            m = grid_nb(grid, m, minus_slot(d));
            if ((unsigned)m >= (unsigned)n_rows) return false;
            st[2 - o] = m;
        }
    }
    return true;
}

__device__ __forceinline__ bool same_bits(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

// Scratch of one face of the k_row_* kernels, element s of column (row -
// first row, direction) at [s * ld]: the Roe scalars, the unit normal, the
// characteristic values, the correction terms, the face states, and the six
// stencil rows (two per double; the first is -1 when the chain leaves the
// table).
enum { RF_BASE = 0, RF_KN = ex::FB_N, RF_POS = RF_KN + 3, RF_NEG = RF_POS + 5, RF_CA = RF_NEG + 5, RF_CB = RF_CA + 5,
       RF_QP = RF_CB + 5, RF_QN = RF_QP + 5, RF_ROWS = RF_QN + 5, RF_N = RF_ROWS + 3 };
static_assert(RF_N == kRowFace, "scratch of a row's face");

struct RowRound {
    double *p;      // [3][RF_N][ld]
    int r0, r1;     // rows of this round
    int ld;
};

__device__ __forceinline__ double *row_column(const RowRound &R, int gid, int d)
{
    return R.p + (size_t)d * RF_N * R.ld + (gid - R.r0);
}

__device__ __forceinline__ void stencil_rows(const double *col, size_t ld, int st[6])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double w = col[(RF_ROWS + k) * ld];
        st[2 * k] = (int)xi::hi32(w);
        st[2 * k + 1] = (int)xi::lo32(w);
    }
}

__global__ void __launch_bounds__(128, 6) k_row_base(const int *__restrict__ grid, const double *__restrict__ metric,
                                                     const double *__restrict__ roe, int n_rows, RowRound R)
{
    const int gid = R.r0 + blockIdx.x * blockDim.x + threadIdx.x, d = blockIdx.y;
    if (gid >= R.r1) return;
    double *col = row_column(R, gid, d);
    const size_t ld = R.ld;
    int st[6];
    if (!plus_line(grid, gid, n_rows, d, st)) {
        col[RF_ROWS * ld] = xi::words(0xffffffffu, 0u);
        return;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) col[(RF_ROWS + k) * ld] = xi::words((uint32_t)st[2 * k], (uint32_t)st[2 * k + 1]);
    const double *fm = metric + 63 * (size_t)gid + 9 * (1 + 2 * d) + 3 * d;
    const double *ra = roe + 36 * (size_t)gid + 6 * d;
    const double r[5] = {ra[0], ra[1], ra[2], ra[4], ra[5]};
    double kn[3], B[ex::FB_N];
    ex::face_normal(fm[0], fm[1], fm[2], kn);
    ex::face_base(r, kn, B);
#pragma unroll
    for (int s = 0; s < ex::FB_N; ++s) col[(RF_BASE + s) * ld] = B[s];
#pragma unroll
    for (int c = 0; c < 3; ++c) col[(RF_KN + c) * ld] = kn[c];
}

// blocks of 256 whose warps keep to one phase (faces_fp64.cu k_face_char): Weno
// on 96^3 rows 4.77 -> 4.74 ms
__global__ void __launch_bounds__(256, 4) k_row_char(const double *__restrict__ Q, double eps, RowRound R)
{
    const int gid = R.r0 + (blockIdx.x / 5u) * blockDim.x + threadIdx.x, d = blockIdx.y, q = blockIdx.x % 5u;
    double *col = row_column(R, gid, d);
    const size_t ld = R.ld;
    int st[6] = {-1, -1, -1, -1, -1, -1};
    if (gid < R.r1) stencil_rows(col, ld, st);
    const bool face = st[0] >= 0;   // the other threads only meet the barriers
    double pos, neg;
    ex::char_pair(
        face,
        [&](double (&L)[5]) {
            ex::left_row(q, [&](int s) { return col[(RF_BASE + s) * ld]; }, [&](int c) { return col[(RF_KN + c) * ld]; }, L);
        },
        [&](int o, int c) { return Q[5 * (size_t)st[o] + c]; }, eps, pos, neg, ex::BlockSync{});
    if (!face) return;
    col[(RF_POS + q) * ld] = pos;
    col[(RF_NEG + q) * ld] = neg;
}

__global__ void __launch_bounds__(256, 3) k_row_back(const double *__restrict__ F, const double *__restrict__ E,
                                                     const double *__restrict__ G, RowRound R)
{
    const int gid = R.r0 + (blockIdx.x / 5u) * blockDim.x + threadIdx.x, d = blockIdx.y, q = blockIdx.x % 5u;
    if (gid >= R.r1) return;
    double *col = row_column(R, gid, d);
    const size_t ld = R.ld;
    int st[6];
    stencil_rows(col, ld, st);
    if (st[0] < 0) return;
    double qp, qn, f[6], ca, cb;
    ex::back_pair(q, [&](int s) { return col[(RF_BASE + s) * ld]; }, [&](int c) { return col[(RF_KN + c) * ld]; },
                  [&](int s) { return col[(RF_POS + s) * ld]; }, [&](int s) { return col[(RF_NEG + s) * ld]; }, qp, qn);
    col[(RF_QP + q) * ld] = qp;
    col[(RF_QN + q) * ld] = qn;
    const double *NF = (d == 0 ? F : (d == 1 ? E : G)) + q;
#pragma unroll
    for (int o = 0; o < 6; ++o) f[o] = NF[5 * (size_t)st[o]];
    ex::correction_terms(f, ca, cb);
    col[(RF_CA + q) * ld] = ca;
    col[(RF_CB + q) * ld] = cb;
}

// Two lanes per face: Fp[(d*5 + c)*n_all + gid]; also p's -1/2 face
// Fm[(d*5 + c)*n_all + p] with stamp[d*n_all + p] = gen for the plus
// neighbour p whose minus neighbour is gid, when p's face data are gid's
// bit for bit.
__global__ void __launch_bounds__(128, 4) k_row_flux(const double *__restrict__ deter, const int *__restrict__ grid,
                                                     const double *__restrict__ metric, const double *__restrict__ roe,
                                                     int n_items, int n_rows, double *__restrict__ Fp,
                                                     double *__restrict__ Fm, unsigned *__restrict__ stamp,
                                                     unsigned gen, long long n_all, RowRound R)
{
    const int t = R.r0 + (blockIdx.x * blockDim.x + threadIdx.x) / 2, d = blockIdx.y, side = threadIdx.x & 1;
    const bool in = t < R.r1;
    const int gid = in ? t : R.r0;
    const double *col = row_column(R, gid, d);
    const size_t ld = R.ld;
    int st[6];
    stencil_rows(col, ld, st);
    const bool face = in && st[0] >= 0;   // the other lanes take part with a face they do not store
    const double *fm = metric + 63 * (size_t)gid + 9 * (1 + 2 * d) + 3 * d;
    double q[5] = {1.0, 0.0, 0.0, 0.0, 2.5}, m[3] = {1.0, 0.0, 0.0}, det = 1.0, Fh[5];
    if (face) {
#pragma unroll
        for (int c = 0; c < 5; ++c) q[c] = col[(RF_QP + 5 * side + c) * ld];
#pragma unroll
        for (int c = 0; c < 3; ++c) m[c] = fm[c];
        det = deter[6 * (size_t)gid + 2 * d];
    }
    ex::llf_lanes(q, m[0], m[1], m[2], det, Fh);
    if (!face) return;
    const int p = st[3];
    bool shared = (unsigned)p < (unsigned)n_items && grid_nb(grid, p, minus_slot(d)) == gid;
    if (shared) {   // p's -1/2 face reads metric block 2+2d, DETERM 2d+1 and ROE block d+3 of p
        const double *mp = metric + 63 * (size_t)p + 9 * (2 + 2 * d) + 3 * d;
        const double *rg = roe + 36 * (size_t)gid + 6 * d, *rp = roe + 36 * (size_t)p + 6 * (d + 3);
        shared = same_bits(m[0], mp[0]) && same_bits(m[1], mp[1]) && same_bits(m[2], mp[2])
                 && same_bits(det, deter[6 * (size_t)p + 2 * d + 1]) && same_bits(rg[0], rp[0])
                 && same_bits(rg[1], rp[1]) && same_bits(rg[2], rp[2]) && same_bits(rg[4], rp[4])
                 && same_bits(rg[5], rp[5]);
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        if ((c >= 3) != (side != 0)) continue;   // components 0..2 on the even lane, 3..4 on the odd one
        const double f = Fh[c] - col[(RF_CA + c) * ld] + col[(RF_CB + c) * ld];
        Fp[(d * 5 + c) * n_all + gid] = f;
        if (shared) Fm[(d * 5 + c) * n_all + p] = f;
    }
    if (shared && side == 0) stamp[d * n_all + p] = gen;
}

// Rows of offsets -3..2 of row n along d; false if the chain leaves
// [0, n_rows).
__device__ __forceinline__ bool minus_line(const int *grid, int n, int n_rows, int d, int st[6])
{
    st[3] = n;
    int m = n, p = n;
#pragma unroll
    for (int o = 1; o <= 3; ++o) {
        m = grid_nb(grid, m, minus_slot(d));
        if ((unsigned)m >= (unsigned)n_rows) return false;
        st[3 - o] = m;
        if (o <= 2) {
            p = grid_nb(grid, p, plus_slot(d));
            if ((unsigned)p >= (unsigned)n_rows) return false;
            st[3 + o] = p;
        }
    }
    return true;
}

// The -1/2 face of every row gid < n_items along each d that the k_row_* kernels
// did not stamp, from the row's own face data (metric block 2+2d, DETERM
// 2d+1, ROE block d+3): Fm and stamp = gen.  A grid-stride scan of the
// rows, direction by direction, with a resident-sized grid: on a periodic
// lattice every face is stamped and the pass only reads the stamps.
__global__ void __launch_bounds__(128, 2) k_weno_minus(Phys P, const double *__restrict__ deter,
                                                        const int *__restrict__ grid, const double *__restrict__ Q,
                                                        const double *__restrict__ metric,
                                                        const double *__restrict__ roe, const double *__restrict__ F,
                                                        const double *__restrict__ E, const double *__restrict__ G,
                                                        int n_items, int n_rows, double *__restrict__ Fm,
                                                        unsigned *__restrict__ stamp, unsigned gen, long long ld)
{
    const int stride = gridDim.x * blockDim.x;
    for (int d = 0; d < 3; ++d) {
        for (int gid = blockIdx.x * blockDim.x + threadIdx.x; gid < n_items; gid += stride) {
            if (stamp[d * ld + gid] == gen) continue;
            int st[6];
            if (!minus_line(grid, gid, n_rows, d, st)) continue;   // k_weno reports the row
            double Fh[5];
            face_side(P, gid, d, 1, st, deter, Q, metric, roe, d == 0 ? F : (d == 1 ? E : G), Fh);
#pragma unroll
            for (int c = 0; c < 5; ++c) Fm[(d * 5 + c) * ld + gid] = Fh[c];
            stamp[d * ld + gid] = gen;
        }
    }
}

// Weno.cl:36-3137: per row, both faces of each direction from the row's own
// face data (metric blocks, DETERM, ROE_AVERAGING), as the reference does.
// REUSE: the +1/2 faces come from the k_row_* kernels (Fp), the -1/2 faces from Fm
// (the k_row_* kernels or k_weno_minus; every row whose stencil stays in the table
// is stamped with this call's generation).
template <bool REUSE>
__global__ void __launch_bounds__(128, REUSE ? 5 : 1) k_weno(Phys P, int j, double mach, double dt, const double *__restrict__ deter,
                                              const double *__restrict__ det, double *__restrict__ U0,
                                              double *__restrict__ U1, double *__restrict__ U2,
                                              const int *__restrict__ grid, const double *__restrict__ Q,
                                              const double *__restrict__ metric, const double *__restrict__ roe,
                                              const double *__restrict__ Fv, const double *__restrict__ Ev,
                                              const double *__restrict__ Gv, const double *__restrict__ F,
                                              const double *__restrict__ E, const double *__restrict__ G,
                                              double *__restrict__ flow, int n_items, int n_rows, unsigned *flags,
                                              double *__restrict__ L_out, const double *__restrict__ Fp,
                                              const double *__restrict__ Fm, const unsigned *__restrict__ stamp,
                                              unsigned gen, long long ld)
{
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n_items) return;
    int idx[3][7];
    if (!gather_star(grid, gid, n_rows, idx)) {
        atomicOr(flags, CFD_FLAG_BAD_INDEX);
        return;
    }
    double dflux[3][5], dvis[3][5];
    bool bad = false;
    // direction d's flux and viscous differences (unrolled over d with the
    // faces from the scratch, a loop when the faces are evaluated here)
    auto direction = [&](const int d) {
        const double *NF = d == 0 ? F : (d == 1 ? E : G);
        const double *VF = d == 0 ? Fv : (d == 1 ? Ev : Gv);
        double Fh[2][5];
        if (REUSE) {
            if (stamp[d * ld + gid] != gen) {   // cannot happen when the star is in the table
                bad = true;
                return;
            }
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                Fh[0][c] = Fp[(d * 5 + c) * ld + gid];
                Fh[1][c] = Fm[(d * 5 + c) * ld + gid];
            }
        } else {
#pragma unroll 1
            for (int s = 0; s < 2; ++s)   // stencil rows: offsets -2..3 (plus) or -3..2 (minus)
                face_side(P, gid, d, s, idx[d] + (s == 0 ? 1 : 0), deter, Q, metric, roe, NF, Fh[s]);
        }
        int Lc[7];
#pragma unroll
        for (int o = 0; o < 7; ++o) Lc[o] = grid_loc(grid, idx[d][o]);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            dflux[d][c] = Fh[0][c] - Fh[1][c];
        }
        const int b = weno_visc_branch(Lc);
        if (b == 5) {
            ex::central4<true>([&](int o, int c) { return VF[5 * (size_t)idx[d][o + 3] + c]; }, dvis[d]);
        } else {
#pragma unroll
            for (int c = 0; c < 5; ++c)
                dvis[d][c] = row_deriv(VF + c, idx[d][0], idx[d][1], idx[d][2], idx[d][3], idx[d][4], idx[d][5],
                                       idx[d][6], b);
        }
    };
    if (REUSE) {
        direction(0);
        direction(1);
        direction(2);
    } else {
#pragma unroll 1
        for (int d = 0; d < 3; ++d) direction(d);
    }
    if (bad) {
        atomicOr(flags, CFD_FLAG_BAD_INDEX);
        return;
    }
    double L[5];
#pragma unroll
    for (int c = 0; c < 5; ++c)
        L[c] = (-1.0) * (dflux[0][c] + dflux[1][c] + dflux[2][c] + dvis[0][c] + dvis[1][c] + dvis[2][c]);
    if (L_out) {
#pragma unroll
        for (int c = 0; c < 5; ++c) L_out[5 * (size_t)gid + c] = L[c];
    }
    // SSP-RK3 stage and primitive recovery (Weno.cl:3084-3135)
    const size_t r5 = 5 * (size_t)gid;
    double u0[5], u1[5], u2[5], Un[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) { u0[c] = U0[r5 + c]; u1[c] = U1[r5 + c]; u2[c] = U2[r5 + c]; }
    double rho, u, v, w, e, p, t, a;
    ex::rk_and_primitives<true>(j, dt, mach, det[gid], u0, u1, u2, L, Un, rho, u, v, w, e, p, t, a);
    double *Uo = j == 0 ? U1 : (j == 1 ? U2 : U0);
#pragma unroll
    for (int c = 0; c < 5; ++c) Uo[r5 + c] = Un[c];
    double *fo = flow + 9 * (size_t)gid;
    fo[FRHO] = rho;
    fo[FU] = u;
    fo[FV] = v;
    fo[FW] = w;
    fo[FE] = e;
    fo[FP] = p;
    fo[FT] = t;
    fo[FA] = a;
    if (gid > 0 && !(isfinite(rho) && isfinite(u) && isfinite(v) && isfinite(w) && isfinite(p)))
        atomicOr(flags, CFD_FLAG_NONFINITE);
}

cudaError_t row_scratch_alloc(RowScratch &S, long long rows)
{
    RowScratch n;
    n.rows = rows;
    n.round = std::min(rows, kRowRound);
    cudaError_t e = cudaMalloc((void **)&n.face, row_face_bytes(rows));
    if (e == cudaSuccess) e = cudaMemset(n.stamps(), 0, (size_t)rows * 3 * sizeof(unsigned));
    if (e == cudaSuccess) e = round_alloc(n.round, std::min(rows, kLeastRound), row_round_bytes, (void **)&n.col);
    if (e != cudaSuccess) {
        cudaGetLastError();
        row_scratch_free(n);
    }
    S = n;
    return e;
}

void row_scratch_free(RowScratch &S)
{
    if (S.face) cudaFree(S.face);
    if (S.col) cudaFree(S.col);
    S = RowScratch();
}

int launch_uq(cudaStream_t st, double *U, double *Q, const int *grid, const double *det, const double *flow,
              double *roe, int n_items, int n_rows, unsigned *flags, const RowScratch &scratch)
{
    if (scratch.serves(n_rows)) {
        k_uq_node<<<blocks_for(n_rows, 128), 128, 0, st>>>(flow, n_rows, scratch.face);
        k_uq<true><<<blocks_for(n_items, 128), 128, 0, st>>>(U, Q, grid, det, flow, roe, n_items, n_rows, flags,
                                                             scratch.face);
        return 2;
    }
    k_uq<false><<<blocks_for(n_items, 128), 128, 0, st>>>(U, Q, grid, det, flow, roe, n_items, n_rows, flags, nullptr);
    return 1;
}

int launch_viscous(cudaStream_t st, const Phys &P, const double *U, double *F, double *E, double *G, double *Fv,
                    double *Ev, double *Gv, const int *grid, const double *metric, const double *det, double *flow,
                    int n_items, int n_rows, unsigned *flags)
{
    const bool fp = n_items <= kPlainNodes;
    const int T = fp ? kViscousThreads<false> : kViscousThreads<true>;
    (fp ? k_node_flux<false> : k_node_flux<true>)<<<blocks_for(n_items, 128), 128, 0, st>>>(
        F, E, G, Fv, grid, metric, det, flow, n_items, n_rows, P.les);
    (fp ? k_viscous<false> : k_viscous<true>)<<<blocks_for(n_items, T), T, 0, st>>>(P, U, Fv, Ev, Gv, grid, metric, det,
                                                                                    flow, n_items, n_rows, flags);
    return 2;
}

// Grid of k_weno_minus: two resident blocks of 128 per SM, at most one
// thread per row.
static unsigned minus_blocks(int n_items)
{
    const long long want = ((long long)n_items + 127) / 128;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess
        || sms <= 0) {
        cudaGetLastError();
        return (unsigned)std::max(1LL, want);
    }
    return (unsigned)std::max(1LL, std::min<long long>(want, 2LL * sms));
}

void launch_weno(cudaStream_t st, const Phys &P, int j, double mach, double dt, const double *deter,
                 const double *det, double *U0, double *U1, double *U2, const int *grid, const double *Q,
                 const double *metric, const double *roe, const double *Fv, const double *Ev, const double *Gv,
                 const double *F, const double *E, const double *G, double *flow, int n_items, int n_rows,
                 unsigned *flags, double *L_out, const RowScratch &scratch, unsigned gen)
{
    const unsigned nb = blocks_for(n_items, 128);
    if (scratch.serves(n_items)) {
        const long long ld = scratch.rows;
        double *Fp = scratch.face, *Fm = scratch.face + 15 * ld;
        unsigned *stamp = scratch.stamps();
        const int round = (int)scratch.round;
        for (int r0 = 0; r0 < n_items; r0 += round) {
            const RowRound R{scratch.col, r0, std::min(n_items, r0 + round), round};
            const unsigned n = blocks_for(R.r1 - r0, 128), n2 = blocks_for(R.r1 - r0, 256);
            k_row_base<<<dim3(n, 3), 128, 0, st>>>(grid, metric, roe, n_rows, R);
            k_row_char<<<dim3(5 * n2, 3), 256, 0, st>>>(Q, P.eps, R);
            k_row_back<<<dim3(5 * n2, 3), 256, 0, st>>>(F, E, G, R);
            k_row_flux<<<dim3(blocks_for(2LL * (R.r1 - r0), 128), 3), 128, 0, st>>>(
                deter, grid, metric, roe, n_items, n_rows, Fp, Fm, stamp, gen, ld, R);
        }
        k_weno_minus<<<minus_blocks(n_items), 128, 0, st>>>(P, deter, grid, Q, metric, roe, F, E, G, n_items, n_rows,
                                                             Fm, stamp, gen, ld);
        k_weno<true><<<nb, 128, 0, st>>>(P, j, mach, dt, deter, det, U0, U1, U2, grid, Q, metric, roe, Fv, Ev, Gv, F, E,
                                         G, flow, n_items, n_rows, flags, L_out, Fp, Fm, stamp, gen, ld);
    } else {
        k_weno<false><<<nb, 128, 0, st>>>(P, j, mach, dt, deter, det, U0, U1, U2, grid, Q, metric, roe, Fv, Ev, Gv, F,
                                          E, G, flow, n_items, n_rows, flags, L_out, nullptr, nullptr, nullptr, 0u, 0);
    }
}

}  // namespace cfd
