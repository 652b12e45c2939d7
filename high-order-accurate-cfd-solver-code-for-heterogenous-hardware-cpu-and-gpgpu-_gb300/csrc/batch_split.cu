// batch_split.cu -- the batched stage (batch_kernel.cuh) instantiated with the
// per-node operations of the split precision form (lattice_split.cuh: FP64
// state, RK3 and face-flux metric products; FP32 characteristic WENO, LLF
// speed and viscous fluxes), compiled with FMA contraction and approximate
// FP32 division/sqrt.
#include "batch_kernel.cuh"
#include "batch_ops.h"
#include "internal.h"
#include "lattice_split.cuh"

namespace cfd {
namespace {

struct Ops {
    static constexpr int kFaceBlocks = 7;   // as the single lattice's face pass
    template <int D, int TILE>
    static __device__ __forceinline__ void face_tile(const LatView &g, TileAt at, float *smem)
    {
        sp::face_tile<FaceTile<D, TILE, true>, D>(g, at, smem);
    }
    static __device__ __forceinline__ void prep(const LatView &g, int n, int q) { sp::init_node(g, n, q); }
    // the viscous pass on the hi/lo read copy of the stage's state
    static __device__ __forceinline__ void visc(const LatView &g, int n, int) { mx::visc_node<false>(sp::hilo_view(g), n, 0); }
    static __device__ __forceinline__ void mu(const LatView &g, int n, int) { mx::mu_node(sp::hilo_view(g), n, 0); }
    static __device__ __forceinline__ void update(const LatView &g, int n, int j) { sp::update_node<false>(g, n, j); }
};

}  // namespace

cudaError_t batch_stage_split(const BatchLaunch &b, int j) { return batch_stage_reduced<Ops>(b, j); }

void batch_prep_split(const LatView &g, cudaStream_t st)
{
    k_batch_prep<Ops><<<blocks_for(g.N, 128), 128, 0, st>>>(g);
}

int batch_occupancy_split(int threads) { return batch_occupancy_reduced<Ops>(threads); }

}  // namespace cfd
