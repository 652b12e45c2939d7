// batch_ops.h -- host-side launch interface of the batched stage for the
// precision forms (batch_fp64.cu, batch_mixed.cu, batch_split.cu).
#pragma once

#include <cuda_runtime.h>

#include "lattice.cuh"

namespace cfd {

struct BatchTile;
struct BatchItem;

// Faces along the direction of the reduced forms' face tiles (kFaceThreads
// faces each, FLAT; face_tile.cuh): along i the width that costs least on an
// instance's extents (batch.cu i_tiles_of), along j and k always the short
// one, whose rows across are whole cache lines.
constexpr int kBatchTilesI[3] = {8, 16, 32};
constexpr int kBatchTileJK = 8;

struct BatchLaunch {
    const LatView *views;      // device table
    const BatchTile *tiles;    // device table
    int ntiles;
    int threads;               // = tile size
    int blocks;                // co-resident persistent grid
    unsigned *bar;             // device barrier words (2)
    unsigned *gflags;          // device error word of the batch
    unsigned long long limit_ns;
    cudaStream_t stream;
    // reduced forms: viscous ranges and face tiles
    const BatchItem *items = nullptr;
    int nitems = 0;
    // FP64 form: the face kernels' scratch, [3][kFaceScratchNormals] columns of
    // round_tiles tiles
    double *scratch = nullptr;
    int round_tiles = 0;
};

// Launches a kernel and returns the launch's own error: an error that other
// code left pending on this thread is neither taken for it nor cleared.
template <class... P, class... A>
cudaError_t batch_launch(void (*kernel)(P...), dim3 grid, int threads, cudaStream_t stream, bool cooperative, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cooperative ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Nodes whose faces one round of the FP64 form's face kernels takes at most
// (1.13 GB of scratch).
constexpr int kBatchRound = 1 << 20;

// One RK stage j (its last or only launch cooperative).  Returns the launch
// error.
cudaError_t batch_stage_fp64(const BatchLaunch &b, int j);
cudaError_t batch_stage_mixed(const BatchLaunch &b, int j);
cudaError_t batch_stage_split(const BatchLaunch &b, int j);
// Launches of one FP64 stage (the reduced forms: 2).
int batch_launches_fp64(int ntiles, int round_tiles);
// Stage-0 prep of one lattice.
void batch_prep_fp64(const LatView &g, cudaStream_t st);
void batch_prep_mixed(const LatView &g, cudaStream_t st);
void batch_prep_split(const LatView &g, cudaStream_t st);
// Co-resident blocks per SM of the closing kernel at `threads` per block.
int batch_occupancy_fp64(int threads);
int batch_occupancy_mixed(int threads);
int batch_occupancy_split(int threads);

}  // namespace cfd
