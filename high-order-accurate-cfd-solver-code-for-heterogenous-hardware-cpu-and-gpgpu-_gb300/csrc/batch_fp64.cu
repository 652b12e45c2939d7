// batch_fp64.cu -- the batched stage in the FP64 form (compiled with
// --fmad=false, reference evaluation order).
//
// The FP64 pipe bounds it, so it runs as the single lattice does
// (faces_fp64.cu): the viscous fluxes and the face pass as kernels of their
// own over the tile table of all instances, each at the registers its part
// needs, and only the last one -- the LLF fluxes, the grid barrier, then the
// update with the next stage's U_Q -- as a persistent cooperative launch.
// One persistent launch for the whole stage needed 250 registers (8 warps
// per SM), too few to hide the integer chains of the products and quotients.
// The face scratch is the batch's, kept between steps, for at most
// kBatchRound nodes and within what the instances leave of the budget; a
// larger batch runs its faces in rounds of tiles.  The unit normals are formed
// into it by each stage instead of kept per instance, so that a budget filled
// to the last instance still has rounds of a fourteenth of the batch.
// 8 vortices (24^3-48^3, 384,631 nodes), one step with FLOW in and out:
// 13.9 ms as one persistent launch per stage, 11.8 with the integer products
// in it, 8.7 ms here.
#include "batch_kernel.cuh"
#include "batch_ops.h"
#include "internal.h"
#include "lattice_fp64.cuh"

namespace cfd {
namespace {

struct Ops {
    static __device__ __forceinline__ void prep(const LatView &g, int n, int q) { ex::prep_node<true>(g, n, q); }
};

__global__ void __launch_bounds__(256, 2) k_batch_visc(const LatView *__restrict__ views,
                                                       const BatchTile *__restrict__ tiles, int jst)
{
    const BatchTile t = tiles[blockIdx.x];
    if ((int)threadIdx.x >= t.count) return;
    const LatView &g = views[t.inst];
    if (g.P.viscous) ex::visc_node<true>(g, t.n0 + threadIdx.x, jst);
    else ex::mu_node(g, t.n0 + threadIdx.x, jst);
}

// Scratch columns of tile w of a round: the round's tiles back to back.
__device__ __forceinline__ FaceScratch tile_scratch(double *p, const BatchTile &t, int w, int ld)
{
    return {p, t.n0 - w * (int)blockDim.x, ld};
}

// Tiles t0 + w of the round that starts at t0; blockIdx.y the direction,
// neighbouring blocks the fields or components of one tile.
__global__ void __launch_bounds__(256, 4) k_batch_base(const LatView *__restrict__ views,
                                                       const BatchTile *__restrict__ tiles, int t0, double *p, int ld)
{
    const int w = blockIdx.x;
    const BatchTile t = tiles[t0 + w];
    if ((int)threadIdx.x < t.count)
        ex::base_node<true>(views[t.inst], tile_scratch(p, t, w, ld), t.n0 + threadIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(256, 4) k_batch_char(const LatView *__restrict__ views,
                                                       const BatchTile *__restrict__ tiles, int t0, double *p, int ld)
{
    const int w = blockIdx.x / 5u;
    const BatchTile t = tiles[t0 + w];
    ex::char_node<true>(views[t.inst], tile_scratch(p, t, w, ld), t.n0 + threadIdx.x, blockIdx.y, blockIdx.x % 5u,
                  (int)threadIdx.x < t.count, ex::BlockSync{});
}

__global__ void __launch_bounds__(256, 3) k_batch_back(const LatView *__restrict__ views,
                                                       const BatchTile *__restrict__ tiles, int t0, double *p, int ld)
{
    const int w = blockIdx.x / 5u;
    const BatchTile t = tiles[t0 + w];
    if ((int)threadIdx.x < t.count)
        ex::back_node<true>(views[t.inst], tile_scratch(p, t, w, ld), t.n0 + threadIdx.x, blockIdx.y, blockIdx.x % 5u);
}

// Half h of tile w's faces along d, two lanes per face.
__device__ __forceinline__ void flux_half(const LatView *__restrict__ views, const BatchTile *__restrict__ tiles,
                                          int t0, int w, int d, int h, double *p, int ld)
{
    const BatchTile t = tiles[t0 + w];
    const int k = h * (int)(blockDim.x / 2) + (int)(threadIdx.x / 2);
    const bool in = k < t.count;
    ex::flux_node<true>(views[t.inst], tile_scratch(p, t, w, ld), t.n0 + (in ? k : 0), d, in);
}

__global__ void __launch_bounds__(256, 2) k_batch_flux(const LatView *__restrict__ views,
                                                       const BatchTile *__restrict__ tiles, int t0, double *p, int ld)
{
    flux_half(views, tiles, t0, blockIdx.x / 2u, blockIdx.y, blockIdx.x % 2u, p, ld);
}

// The last round's fluxes, the grid barrier, and the update of every tile.
__global__ void __launch_bounds__(256, 2)
k_batch_close(const LatView *__restrict__ views, const BatchTile *__restrict__ tiles, int ntiles, int t0, int jst,
              double *p, int ld, unsigned *bar, unsigned *gflags, unsigned long long limit_ns)
{
    const int items = 6 * (ntiles - t0);
    for (int w = next_item(bar); w < items; w = next_item(bar)) flux_half(views, tiles, t0, w / 6, (w % 6) >> 1, w & 1, p, ld);
    if (!grid_barrier(bar, gridDim.x, limit_ns, gflags)) return;
    for (int w = blockIdx.x; w < ntiles; w += gridDim.x) {
        const BatchTile t = tiles[w];
        if ((int)threadIdx.x < t.count) ex::update_node<true>(views[t.inst], t.n0 + threadIdx.x, jst, true);
    }
}

}  // namespace

cudaError_t batch_stage_fp64(const BatchLaunch &b, int j)
{
    const int T = b.threads, ld = b.round_tiles * T;
    cudaError_t e = cudaSuccess;
    auto launch = [&](auto kernel, dim3 grid, auto... args) {
        if (e == cudaSuccess) e = batch_launch(kernel, grid, T, b.stream, false, b.views, b.tiles, args...);
    };
    launch(k_batch_visc, b.ntiles, j);
    int t0 = 0;
    for (;; t0 += b.round_tiles) {
        const int nt = b.ntiles - t0 < b.round_tiles ? b.ntiles - t0 : b.round_tiles;
        launch(k_batch_base, dim3(nt, 3), t0, b.scratch, ld);
        launch(k_batch_char, dim3(5 * nt, 3), t0, b.scratch, ld);
        launch(k_batch_back, dim3(5 * nt, 3), t0, b.scratch, ld);
        if (t0 + nt == b.ntiles) break;   // the closing launch takes this round's fluxes
        launch(k_batch_flux, dim3(2 * nt, 3), t0, b.scratch, ld);
    }
    if (e != cudaSuccess) return e;
    return batch_launch(k_batch_close, b.blocks, T, b.stream, true, b.views, b.tiles, b.ntiles, t0, j, b.scratch, ld, b.bar,
                        b.gflags, b.limit_ns);
}

int batch_launches_fp64(int ntiles, int round_tiles)
{
    const int rounds = (ntiles + round_tiles - 1) / round_tiles;
    return 1 + 4 * rounds;   // viscous; base, char, back and the fluxes or the closing launch
}

void batch_prep_fp64(const LatView &g, cudaStream_t st)
{
    k_batch_prep<Ops><<<blocks_for(g.N, 128), 128, 0, st>>>(g);
}

int batch_occupancy_fp64(int threads)
{
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_batch_close, threads, 0) != cudaSuccess) return 0;
    return nb;
}

}  // namespace cfd
