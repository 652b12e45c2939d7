// face_tile.cuh -- shared-memory tiles of the FP32 face passes (mixed and
// split forms): a block of 128 threads covers TILE faces along the face
// direction D times 128 / TILE nodes across it (axis A), on one line of the
// third axis (B).  The block loads the stencil lines (TILE + 5 nodes along
// D) of Q, the Roe inputs (u, v, w, sqrt(rho), H) and the node fluxes along
// D once, coalesced along i, and every face reads its six points from there
// (the reference gathers each point per face, Weno.cl:159-328).
#pragma once

#include "lattice.cuh"
#include "physics.cuh"

namespace cfd {

constexpr int kFaceThreads = 128;

// FLAT: the nodes across are consecutive nodes of the plane across D (axis A
// fastest) instead of a piece of one line, so that only the extent along D
// pads a tile: for small lattices.
template <int D, int TILE, bool FLAT = false>
struct FaceTile {
    static constexpr bool kFlat = FLAT;
    static constexpr int kTile = TILE;                   // faces along D
    static constexpr int kWide = kFaceThreads / TILE;    // nodes across
    static constexpr int A = D == 0 ? 1 : 0;             // axis across
    static constexpr int B = D == 2 ? 1 : 2;             // axis of the block's line
    static constexpr int kLine = kTile + 5;              // staged nodes along D
    static constexpr int kStaged = kLine * kWide;
    // smem index of (position b along D, a across); i is the fast index
    static __device__ __forceinline__ int at(int b, int a) { return D == 0 ? a * kLine + b : b * kWide + a; }
    // thread -> (t along D, a across), consecutive threads consecutive in i
    static __device__ __forceinline__ void split(int x, int &t, int &a)
    {
        if (D == 0) {
            t = x % kTile;
            a = x / kTile;
        } else {
            t = x / kWide;
            a = x % kWide;
        }
    }
    // staged element m -> (b along D, a across)
    static __device__ __forceinline__ void staged(int m, int &b, int &a)
    {
        if (D == 0) {
            b = m % kLine;
            a = m / kLine;
        } else {
            b = m / kWide;
            a = m % kWide;
        }
    }
    static dim3 grid(const LatView &g)
    {
        if (FLAT)
            return dim3((unsigned)((lat_extent_h(g, D) + kTile - 1) / kTile),
                        (unsigned)((g.N / lat_extent_h(g, D) + kWide - 1) / kWide), 1u);
        return dim3((unsigned)((lat_extent_h(g, D) + kTile - 1) / kTile),
                    (unsigned)((lat_extent_h(g, A) + kWide - 1) / kWide), (unsigned)lat_extent_h(g, B));
    }
};

// coordinate c in [-2, n + TILE + 3) of a staged stencil line, wrapped
// (periodic) or clamped; the wrap subtracts instead of dividing (c is at
// most a few extents away from [0, n))
__device__ __forceinline__ int tile_coord(const LatView &g, int d, int c)
{
    const int n = lat_extent(g, d);
    if (lat_periodic(g, d)) {
        while (c < 0) c += n;
        while (c >= n) c -= n;
        return c;
    }
    return c < 0 ? 0 : (c >= n ? n - 1 : c);
}

// The node of plane index m (FLAT tiles) at coordinate cD along D.
template <int D>
__device__ __forceinline__ int plane_node(const LatView &g, int m, int cD)
{
    if (D == 0) return cD + g.ni * m;
    if (D == 2) return m + g.ni * g.nj * cD;
    const int k = (int)((unsigned)m / (unsigned)g.ni);
    return m - g.ni * k + g.ni * (cD + g.nj * k);
}

// The tile at face coordinate tD along D, node tA across (axis A, or of the
// plane), line cB of axis B: the single-lattice passes take it from blockIdx, the batched
// kernel from its item table.
struct TileAt {
    int tD, tA, cB;
};

// The tile of block w of T's grid (gr) laid out in one dimension.
template <class T>
__device__ __forceinline__ TileAt tile_of_index(unsigned w, uint3 gr)
{
    const unsigned r = w / gr.x;
    return {(int)(w - r * gr.x) * T::kTile, (int)(r % gr.y) * T::kWide, (int)(r / gr.y)};
}

template <class T>
__device__ __forceinline__ TileAt tile_of_block()
{
    return {(int)blockIdx.x * T::kTile, (int)blockIdx.y * T::kWide, (int)blockIdx.z};
}

// What derive left of a node that its flux along D takes: rho from Q, the
// velocities from the Roe inputs, the pressure, the node metrics.  Forming
// the flux where it is read (at most 1.6 times per face) takes 15 loads and
// 15 stores per node out of the update and 60 bytes per node out of memory.
struct NodeIn {
    float prim[5], m[3], det;
};
template <int D>
__device__ __forceinline__ NodeIn lat_node_in(const LatView &g, int node)
{
    const int N = g.N;
    return {{__ldg(g.Q32 + node), __ldg(g.R32 + node), __ldg(g.R32 + N + node), __ldg(g.R32 + 2 * N + node),
             __ldg(g.prim32 + LF_P * N + node)},
            {__ldg(g.node32 + 3 * D * N + node), __ldg(g.node32 + (3 * D + 1) * N + node),
             __ldg(g.node32 + (3 * D + 2) * N + node)},
            __ldg(g.node32 + 9 * N + node)};
}

// Stages the block's stencil lines of Q, the Roe inputs and the node fluxes
// along D (read-only in the face pass: non-coherent loads) into sQ/sR/sF, each
// [5][T::kStaged]; ends with __syncthreads().  A block stages 1.04 to 1.6
// nodes per thread: all of a thread's loads are issued before its first
// store, so that the block waits for memory once (a direction of
// TGV 128^3, split: 0.100 -> 0.097 ms).
template <class T, int D>
__device__ __forceinline__ void stage_face_lines(const LatView &g, TileAt at, float *sQ, float *sR, float *sF)
{
    constexpr int S = T::kStaged, R = (S + kFaceThreads - 1) / kFaceThreads;
    const int N = g.N;
    const int nA = T::kFlat ? lat_extent(g, T::A) * lat_extent(g, T::B) : lat_extent(g, T::A);
    int e[R];
    NodeIn in[R];
    float q[R][4], r[R][2];   // Q past rho, the Roe inputs past the velocities
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int m = threadIdx.x + k * kFaceThreads;
        if (k == R - 1 && m >= S) break;
        int b, a;
        T::staged(m, b, a);
        const int cD = tile_coord(g, D, at.tD + b - 2), cA = at.tA + a < nA ? at.tA + a : nA - 1;
        int node;
        if (T::kFlat) {
            node = plane_node<D>(g, cA, cD);
        } else {
            int c[3];
            c[D] = cD;
            c[T::A] = cA;
            c[T::B] = at.cB;
            node = c[0] + g.ni * (c[1] + g.nj * c[2]);
        }
        e[k] = T::at(b, a);
        in[k] = lat_node_in<D>(g, node);
#pragma unroll
        for (int x = 0; x < 4; ++x) q[k][x] = __ldg(g.Q32 + (x + 1) * N + node);
#pragma unroll
        for (int x = 0; x < 2; ++x) r[k][x] = __ldg(g.R32 + (x + 3) * N + node);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        if (k == R - 1 && (int)threadIdx.x + k * kFaceThreads >= S) break;
        float f[5];
        node_inviscid_flux(in[k].prim, in[k].m, in[k].det, f);
        sQ[e[k]] = in[k].prim[0];
#pragma unroll
        for (int x = 0; x < 4; ++x) sQ[(x + 1) * S + e[k]] = q[k][x];
#pragma unroll
        for (int x = 0; x < 3; ++x) sR[x * S + e[k]] = in[k].prim[x + 1];
#pragma unroll
        for (int x = 0; x < 2; ++x) sR[(x + 3) * S + e[k]] = r[k][x];
#pragma unroll
        for (int x = 0; x < 5; ++x) sF[x * S + e[k]] = f[x];
    }
    __syncthreads();
}

// The face of this thread: its lattice node and position (t, a) in the
// tile; false if the thread has no face (past the lattice, or a face whose
// stencil leaves a non-periodic box).
template <class T, int D>
__device__ __forceinline__ bool tile_face(const LatView &g, TileAt at, int &n, int &t, int &a)
{
    T::split(threadIdx.x, t, a);
    int c[3];
    c[D] = at.tD + t;
    if (T::kFlat) {
        c[T::A] = c[T::B] = 0;
        if (c[D] >= lat_extent(g, D) || at.tA + a >= lat_extent(g, T::A) * lat_extent(g, T::B)
            || !lat_face_needed(g, c[0], c[1], c[2], D))
            return false;
        n = plane_node<D>(g, at.tA + a, c[D]);
        return true;
    }
    c[T::A] = at.tA + a;
    c[T::B] = at.cB;
    if (c[D] >= lat_extent(g, D) || c[T::A] >= lat_extent(g, T::A) || !lat_face_needed(g, c[0], c[1], c[2], D))
        return false;
    n = c[0] + g.ni * (c[1] + g.nj * c[2]);
    return true;
}

// The stencil of the face at tile position (t, a) from the staged lines:
// P[k] = (Q of point k, Q of point 5-k) and the Roe state r of the face.
template <class T>
__device__ __forceinline__ void tile_stencil(const float *sQ, const float *sR, int t, int a, float2 P[3][5],
                                             float r[5])
{
    constexpr int S = T::kStaged;
#pragma unroll
    for (int o = 0; o < 3; ++o)
#pragma unroll
        for (int q = 0; q < 5; ++q) P[o][q] = make_float2(sQ[q * S + T::at(t + o, a)], sQ[q * S + T::at(t + 5 - o, a)]);
    const int er = T::at(t + 3, a), el = T::at(t + 2, a);
    roe_average(sR[3 * S + er], sR[er], sR[S + er], sR[2 * S + er], sR[4 * S + er], sR[3 * S + el], sR[el],
                       sR[S + el], sR[2 * S + el], sR[4 * S + el], r);
}

// The node fluxes f[0..5] of component q along D at tile position (t, a).
template <class T>
__device__ __forceinline__ void tile_node_fluxes(const float *sF, int q, int t, int a, float f[6])
{
    constexpr int S = T::kStaged;
#pragma unroll
    for (int o = 0; o < 6; ++o) f[o] = sF[q * S + T::at(t + o, a)];
}

// Shared floats one tile of T stages (Q, Roe inputs, node fluxes).
template <class T>
constexpr int tile_smem_floats()
{
    return 15 * T::kStaged;
}

// A stage's fluxes in one launch: blocks 0 .. nv - 1 a viscous range each
// (their chains are the longest), then the face tiles along i, j and k.
// Ops::visc<LOC>(g, n, q) and Ops::face_tile<T, D>(g, at, smem) of one form.
struct FluxGrid {
    unsigned nv, b[2];   // viscous ranges; end of the i tiles, of the j tiles
    uint3 gr[3];
};
// Small and odd extents: FLAT tiles of 16 and 8 (split 33^3 24.9 us a stage,
// 37 x 41 x 19 inviscid 20.7; 27.0 and 22.5 with lines of 32 and 16).
using FluxTileI = FaceTile<0, 16, true>;
using FluxTileJ = FaceTile<1, 8, true>;
using FluxTileK = FaceTile<2, 8, true>;

inline unsigned flux_grid(const LatView &g, FluxGrid &f)
{
    const dim3 d[3] = {FluxTileI::grid(g), FluxTileJ::grid(g), FluxTileK::grid(g)};
    unsigned n = f.nv = (unsigned)((g.N + kFaceThreads - 1) / kFaceThreads);
    for (int k = 0; k < 3; ++k) {
        f.gr[k] = make_uint3(d[k].x, d[k].y, d[k].z);
        n += d[k].x * d[k].y * d[k].z;
        if (k < 2) f.b[k] = n;
    }
    return n;
}

template <class Ops, bool LOC>
__device__ __forceinline__ void flux_block(const LatView &g, int q, const FluxGrid &f, float *smem)
{
    const unsigned w = blockIdx.x;
    if (w < f.nv) {
        const int n = (int)(w * kFaceThreads + threadIdx.x);
        if (n < g.N) Ops::template visc<LOC>(g, n, q);
    } else if (w < f.b[0]) {
        Ops::template face_tile<FluxTileI, 0>(g, tile_of_index<FluxTileI>(w - f.nv, f.gr[0]), smem);
    } else if (w < f.b[1]) {
        Ops::template face_tile<FluxTileJ, 1>(g, tile_of_index<FluxTileJ>(w - f.b[0], f.gr[1]), smem);
    } else {
        Ops::template face_tile<FluxTileK, 2>(g, tile_of_index<FluxTileK>(w - f.b[1], f.gr[2]), smem);
    }
}

constexpr int flux_smem_floats()
{
    constexpr int i = tile_smem_floats<FluxTileI>(), j = tile_smem_floats<FluxTileJ>();
    return i > j ? i : j;
}

// Nodes up to which a reduced form's fluxes run in one launch instead of as
// four kernels on four streams (split form, a stage; four streams against one
// launch): 17^3 nodes 23.2 and 17.1 us, 24^3 23.0 and 20.7, 33^3 29.2 and
// 24.9, 46^3 40.6 and 38.0; 64^3 82.6 and 81.3 (with tiles of 32 and 16), 256
// x 64 x 16 with ghost layers 106 and 113, where each kernel's own registers
// and the tuned tiles tell.
#ifndef CFD_ONE_LAUNCH_NODES
#define CFD_ONE_LAUNCH_NODES 200000
#endif
constexpr int kOneLaunchNodes = CFD_ONE_LAUNCH_NODES;

}  // namespace cfd
