// structured.cu -- face-based RHS kernels for an (i,j,k) lattice, FP64 form.
//
// When the reference's neighbour table is a lattice -- periodic, or padded by
// ghost layers in non-periodic directions (detected by the solver at create
// time, lattice_host.h) -- the same arithmetic runs on a structure-of-arrays
// layout with index arithmetic instead of neighbour chains, and every face is
// computed once.  The reference computes each face twice: as i+1/2 of node i
// and as i-1/2 of node i+1, from identical inputs (the face metric and face
// det of Main.cpp:2369-2440 are single-valued, the Roe average is symmetric
// in its two nodes), so one evaluation per face gives the same fluxes.
//
// Per RK stage j:
//   k_prep    pointwise: Q, U_j = det*Q (U_Q.cl), contravariant node fluxes
//             F,E,G (Viscous.cl:560-631), sqrt(rho) and H for the Roe average
//   k_visc    radius-2 star: viscous + MTS SGS fluxes Fv,Ev,Gv and mu
//   k_face_*  the faces i+1/2 along each direction (faces_fp64.cu): Roe
//             eigenvectors, WENO5, LLF, 6th-order correction -> corrected
//             face flux
//   k_update  pointwise + radius-2: L = -(flux differences + viscous
//             divergence), SSP-RK3 stage j, primitive recovery
// Layout: every field is [component][N] with n = i + ni*(j + nj*k).
//
// The per-node operations live in lattice_fp64.cuh (exact evaluation order)
// and this file is compiled with --fmad=false: the face flux of face i+1/2 is
// bit-identical to what the reference computes for it (twice).  The mixed
// form lives in mixed.cu.
#include "internal.h"
#include "lattice_fp64.cuh"
#include "structured.h"

namespace cfd {

namespace {

__device__ __forceinline__ int node_id() { return blockIdx.x * blockDim.x + threadIdx.x; }

// Blocks of 128 per SM (registers 80, 128, 72): the integer chains of the
// products want warps, the spills cost less.  TGV 128^3: prep 0.31 ms at 4
// to 6 blocks, 0.34 at 8; viscous 1.54 ms at 4, 1.87 at 3, 2.10 at 5;
// update 0.58, 0.54, 0.53, 0.52 ms at 5, 6, 7, 8.  With the products on the
// FP64 pipe they took 0.59, 1.89 and 0.66 ms.
template <bool I>
__global__ void __launch_bounds__(128, 6) k_prep(LatView g, int q)
{
    const int n = node_id();
    if (n < g.N) ex::prep_node<I>(g, n, q);
}

// Blocks of 256 share the integer form's long code better (128^3 1.45 -> 1.33
// ms; 1.44 with barriers between its loops' passes); the plain form's lattices are too small to fill the SMs with them
// (53,000 nodes 0.059 -> 0.073).
template <bool I>
constexpr int kViscThreads = I ? 256 : 128;

template <bool I>
__global__ void __launch_bounds__(kViscThreads<I>, 512 / kViscThreads<I>) k_visc(LatView g, int q)
{
    const int n = node_id();
    if (n < g.N) ex::visc_node<I>(g, n, q);
}

__global__ void __launch_bounds__(128) k_mu_only(LatView g, int q)
{
    const int n = node_id();
    if (n < g.N) ex::mu_node(g, n, q);
}


template <bool I>
__global__ void __launch_bounds__(128, I ? 7 : 4) k_update(LatView g, int jst)
{
    const int n = node_id();
    if (n < g.N) ex::update_node<I>(g, n, jst, false);
}

// AoS reference rows (row stride `stride` doubles) <-> SoA [comp][N].
__global__ void k_aos_to_soa(const double *__restrict__ aos, int stride, int ncomp, long long N,
                             double *__restrict__ soa, const int *__restrict__ row_of)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * ncomp) return;
    const long long n = t / ncomp;
    const int c = (int)(t % ncomp);
    const long long r = row_of ? (long long)row_of[n] : n + 1;
    soa[c * N + n] = aos[r * stride + c];
}

__global__ void k_soa_to_aos(const double *__restrict__ soa, int stride, int ncomp, long long N,
                             double *__restrict__ aos, const int *__restrict__ row_of)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * ncomp) return;
    const long long n = t / ncomp;
    const int c = (int)(t % ncomp);
    const long long r = row_of ? (long long)row_of[n] : n + 1;
    aos[r * stride + c] = soa[c * N + n];
}

}  // namespace

int structured_stage(const StructuredLaunch &S, int jst, double dt, double *Lout, cudaEvent_t *ev,
                     const char **names, int prep_from)
{
    if (S.mixed == 2) return split_stage(S, jst, dt, Lout, ev, prep_from, names);
    if (S.mixed) return mixed_stage(S, jst, dt, Lout, ev, prep_from, names);
    const LatView g = make_view(S, dt, Lout);
    const unsigned nb = blocks_for(g.N, 128);
    cudaStream_t st = S.stream;
    int e = 0, k = 0, entries = 0;
    auto mark = [&](const char *name) {
        if (names) names[entries] = name;
        ++entries;
        if (ev) cudaEventRecord(ev[++e], st);
    };
    if (ev) cudaEventRecord(ev[0], st);
    const bool fp = g.N <= kPlainNodes;   // products of the per-node kernels on the FP64 pipe
    (fp ? k_prep<false> : k_prep<true>)<<<nb, 128, 0, st>>>(g, jst);
    mark("prep");
    // The viscous and the face kernels are independent (the update reads
    // both): side by side the one's latency hides behind the other's work.
    // A stage on 17^3 nodes 107 -> 86 us, 24^3 155 -> 134, 46^3 675 -> 645,
    // 128^3 12.43 -> 12.41 ms.  Not when each launch is timed.
    const bool side = S.side && !ev;
    cudaStream_t sv = side ? S.side : st;
    if (side) {
        cudaEventRecord(S.fork, st);
        cudaStreamWaitEvent(sv, S.fork, 0);
    }
    if (S.P.viscous)
        fp ? k_visc<false><<<blocks_for(g.N, kViscThreads<false>), kViscThreads<false>, 0, sv>>>(g, jst)
           : k_visc<true><<<blocks_for(g.N, kViscThreads<true>), kViscThreads<true>, 0, sv>>>(g, jst);
    else
        k_mu_only<<<nb, 128, 0, sv>>>(g, jst);
    if (side) cudaEventRecord(S.join, sv);
    mark(S.P.viscous ? "viscous" : "mu_only");
    k = 3 + fp64_faces(S, g, st, mark);
    if (side) cudaStreamWaitEvent(st, S.join, 0);
    (fp ? k_update<false> : k_update<true>)<<<nb, 128, 0, st>>>(g, jst);
    mark("update");
    return ev ? entries : k;
}

void aos_to_soa(cudaStream_t st, const double *aos, int stride, int ncomp, long long N, double *soa, const int *row_of)
{
    const long long t = N * ncomp;
    k_aos_to_soa<<<blocks_for(t, 256), 256, 0, st>>>(aos, stride, ncomp, N, soa, row_of);
}

void soa_to_aos(cudaStream_t st, const double *soa, int stride, int ncomp, long long N, double *aos, const int *row_of)
{
    const long long t = N * ncomp;
    k_soa_to_aos<<<blocks_for(t, 256), 256, 0, st>>>(soa, stride, ncomp, N, aos, row_of);
}

}  // namespace cfd
