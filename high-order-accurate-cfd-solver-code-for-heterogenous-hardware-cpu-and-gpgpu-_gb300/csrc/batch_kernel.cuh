// batch_kernel.cuh -- the batched RK stage over many lattices.
//
// Work is described by tables: node tile t = (instance, first node, node
// count), tile size = block size, so one thread owns one node of a tile; and
// (reduced forms) face tiles (face_tile.cuh) of every instance.  A reduced
// form's stage is two launches:
//   k_batch_fluxes          the viscous fluxes (one block per node range) and
//                           the three face fluxes (one block per face tile)
//   k_batch_close_reduced   persistent: the grid-wide barrier, then every
//                           node tile's RHS, RK stage and next U_Q
// (batch_fp64.cu has the FP64 form's launches.)  The closing kernel is
// launched cooperatively (all blocks co-resident) with at most the occupancy
// limit of blocks; the barrier's wait is bounded by a %globaltimer deadline,
// after which it sets CFD_FLAG_TIMEOUT and the block returns instead of
// spinning.
//
// Ops supplies the per-node operations of one precision form
// (lattice_mixed.cuh, lattice_split.cuh); this header is included by the
// translation unit compiled with that form's flags.
#pragma once

#include "batch_ops.h"
#include "face_tile.cuh"
#include "lattice.cuh"

namespace cfd {

struct BatchTile {
    int inst;   // index into the LatView table
    int n0;     // first node of the tile
    int count;  // nodes in the tile (<= block size)
    int pad;
};

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Sense-reversing grid barrier over `nblocks` co-resident blocks.
// bar[0] = arrival count, bar[1] = generation.  Returns false (and sets the
// timeout bit) if the generation does not advance before the deadline.
// The last block to arrive also clears bar[3], the work counter
// (every block has stopped taking items when it arrives), so the
// next launch starts from item 0.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned nblocks, unsigned long long limit_ns,
                                             unsigned *gflags)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        volatile unsigned *vgen = bar + 1;
        const unsigned gen = *vgen;
        __threadfence();
        const unsigned arrived = atomicAdd(bar, 1u);
        if (arrived == nblocks - 1) {
            atomicExch(bar + 3, 0u);
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            const unsigned long long t0 = global_ns();
            while (*vgen == gen) {
                if (global_ns() - t0 > limit_ns) {
                    atomicOr(gflags, 4u);   // CFD_FLAG_TIMEOUT
                    ok = 0;
                    break;
                }
                __nanosleep(200);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Next item before the barrier of this block: blocks take items in order from a
// shared counter (bar[3]), so a block that finishes early takes more and
// no block idles long at the barrier (with a fixed item-to-block map some
// blocks ran ~10 % longer than the rest and everyone waited).
__device__ __forceinline__ int next_item(unsigned *bar)
{
    __shared__ int s_w;
    __syncthreads();   // every thread is done with the previous item
    if (threadIdx.x == 0) s_w = (int)atomicAdd(bar + 3, 1u);
    __syncthreads();
    return s_w;
}

// Kind kBatchVisc: the viscous range of b nodes from node a of one lattice;
// otherwise a face tile (a = first face along its direction, b = first node
// of the plane across): kinds 0 to 2 along i of width kBatchTilesI[kind],
// kinds 3 and 4 along j and k.
constexpr int kBatchVisc = 5;
struct BatchItem {
    int inst, kind, a, b;
};

// The fluxes of every instance: the viscous ranges first (their chains are
// the longest), then the face tiles, one direction after the other's (blocks
// that run at the same time work on one direction's code).  A kernel of its
// own runs at the registers of the
// face pass alone (72); in one persistent launch with the viscous and update
// code it had 80 with spills.  24 vortices of 24^3 to 72^3 (2.7 million
// nodes), a stage: mixed 0.60 -> 0.50 ms, split 0.81 -> 0.79 (0.47 and 0.75
// with FLAT tiles); one of 24^3,
// viscous, mixed 17.3 -> 15.8 us (18.1 with the viscous ranges in the closing
// launch).
template <class Ops>
__global__ void __launch_bounds__(kFaceThreads, Ops::kFaceBlocks)
k_batch_fluxes(const LatView *__restrict__ views, const BatchItem *__restrict__ items, int jst)
{
    __shared__ float smem[tile_smem_floats<FaceTile<0, kBatchTilesI[0]>>()];   // the widest staging
    const BatchItem it = items[blockIdx.x];
    const LatView &g = views[it.inst];
    const TileAt at{it.a, it.b, 0};
    switch (it.kind) {
    case kBatchVisc: {
        if ((int)threadIdx.x >= it.b) return;
        const int n = it.a + threadIdx.x;
        if (g.P.viscous) Ops::visc(g, n, jst);
        else Ops::mu(g, n, jst);
        break;
    }
    case 0: Ops::template face_tile<0, kBatchTilesI[0]>(g, at, smem); break;
    case 1: Ops::template face_tile<0, kBatchTilesI[1]>(g, at, smem); break;
    case 2: Ops::template face_tile<0, kBatchTilesI[2]>(g, at, smem); break;
    case 3: Ops::template face_tile<1, kBatchTileJK>(g, at, smem); break;
    default: Ops::template face_tile<2, kBatchTileJK>(g, at, smem); break;
    }
}

// The grid barrier and the update of every node tile, in blocks of up to 256
// threads (the tile sizes 32, 64, 128, 256) at 64 registers, as the single
// lattice's update.  The barrier orders nothing here (the fluxes are an
// earlier launch's); it is the bounded wait that cfd_batch_set_wait_limit
// sets and that a step reports as CFD_ETIMEOUT when the grid is not
// co-resident, and costs 2 us.
template <class Ops>
__global__ void __launch_bounds__(256, 4)
k_batch_close_reduced(const LatView *__restrict__ views, const BatchTile *__restrict__ tiles, int ntiles, int jst,
                      unsigned *bar, unsigned *gflags, unsigned long long limit_ns)
{
    if (!grid_barrier(bar, gridDim.x, limit_ns, gflags)) return;
    for (int w = blockIdx.x; w < ntiles; w += gridDim.x) {
        const BatchTile t = tiles[w];
        if ((int)threadIdx.x < t.count) Ops::update(views[t.inst], t.n0 + threadIdx.x, jst);
    }
}

// One stage of a reduced form on b.stream.
template <class Ops>
cudaError_t batch_stage_reduced(const BatchLaunch &b, int j)
{
    const cudaError_t e = batch_launch(k_batch_fluxes<Ops>, b.nitems, kFaceThreads, b.stream, false, b.views, b.items, j);
    if (e != cudaSuccess) return e;
    return batch_launch(k_batch_close_reduced<Ops>, b.blocks, b.threads, b.stream, true, b.views, b.tiles, b.ntiles, j, b.bar,
                        b.gflags, b.limit_ns);
}

template <class Ops>
int batch_occupancy_reduced(int threads)
{
    int nb = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_batch_close_reduced<Ops>, threads, 0) == cudaSuccess ? nb : 0;
}

// prep (U_Q) of stage 0 for one lattice, before its first stage
template <class Ops>
__global__ void k_batch_prep(LatView g)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < g.N) Ops::prep(g, n, 0);
}

}  // namespace cfd
