// batch_mixed.cu -- the batched stage (batch_kernel.cuh) instantiated with the
// per-node operations of the mixed precision (FMA contraction, approximate FP32 division/sqrt) form.
#include "batch_kernel.cuh"
#include "batch_ops.h"
#include "internal.h"
#include "lattice_mixed.cuh"

namespace cfd {
namespace {

struct Ops {
    static constexpr int kFaceBlocks = 7;   // as the single lattice's face pass
    template <int D, int TILE>
    static __device__ __forceinline__ void face_tile(const LatView &g, TileAt at, float *smem)
    {
        mx::face_tile<FaceTile<D, TILE, true>, D>(g, at, smem);
    }
    static __device__ __forceinline__ void prep(const LatView &g, int n, int q) { mx::init_node(g, n, q); }
    static __device__ __forceinline__ void visc(const LatView &g, int n, int q) { mx::visc_node<false>(g, n, q); }
    static __device__ __forceinline__ void mu(const LatView &g, int n, int q) { mx::mu_node(g, n, q); }
    static __device__ __forceinline__ void update(const LatView &g, int n, int j) { mx::update_node<false>(g, n, j); }
};

}  // namespace

cudaError_t batch_stage_mixed(const BatchLaunch &b, int j) { return batch_stage_reduced<Ops>(b, j); }

void batch_prep_mixed(const LatView &g, cudaStream_t st)
{
    k_batch_prep<Ops><<<blocks_for(g.N, 128), 128, 0, st>>>(g);
}

int batch_occupancy_mixed(int threads) { return batch_occupancy_reduced<Ops>(threads); }

}  // namespace cfd
