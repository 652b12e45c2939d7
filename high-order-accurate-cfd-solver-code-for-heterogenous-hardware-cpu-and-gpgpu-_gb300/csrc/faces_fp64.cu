// faces_fp64.cu -- the FP64 face pass of a lattice: the faces n+1/2 along i,
// j and k (blockIdx.y) in four kernels (lattice_fp64.cuh), one thread per
//   k_face_base   face: Roe average and the scalars of its eigenvectors
//   k_face_char   face and characteristic field: projection and WENO5 pair
//   k_face_back   face and component: back-projection, 6th-order correction
//   k_face_flux   face and side (two lanes per face): fluxes, LLF
//
// What bounds it: the FP64 pipe, which takes an instruction of a warp every
// 64 clocks per scheduler.  The reference's sums have to run there; its
// products, quotients and roots run on the integer pipe (exact_int.cuh, the
// same bits).  An integer product is a chain of some 25 instructions, so
// that only pays with many warps in flight, and one thread holding a whole
// face's flux needs 200 registers; split into five fields, five components
// and two sides the same work fits 54 to 128 registers (16 to 32 warps per
// SM).  The hand-over between the kernels (kFaceScratch doubles per face)
// costs 0.7 KB per face of L2 and HBM traffic, which the FP64-bound kernels
// hide.  TGV 128^3, all three directions: 16.1 ms with one kernel per
// direction and only the divisions on the integer pipe; 9.9 ms here
// (base 0.30, char 5.88, back 1.97, flux 1.70; the FP64 pipe is busy 65 to
// 80 % of the time, with branch-free groups and an instruction footprint
// that stays near the instruction cache's size as the remaining limits).
#include "internal.h"
#include "lattice_fp64.cuh"
#include "structured.h"

namespace cfd {
namespace {

__global__ void __launch_bounds__(128) k_geometry(LatView g, double *kn, double *del)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < g.N) ex::geometry_node(g, kn, del, n, blockIdx.y);
}

__global__ void __launch_bounds__(128, 6) k_face_base(LatView g, FaceScratch fs, int n1)
{
    const int n = fs.n0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (n < n1) ex::base_node(g, fs, n, blockIdx.y);
}

// MB: the blocks of 256 per SM its registers allow (StructuredLaunch::
// face_mb): 128, 80 or 64 registers.  TGV 128^3 6.5, 6.3, 6.2 ms with blocks
// of 128; vortex 64^3 1.17, 1.10, 1.09 ms; 53,000 ghosted nodes 0.195, 0.184,
// 0.182 ms.  Instruction fetch is what costs it most after the FP64 pipe:
// blocks of 256 instead of 128 at 64 registers 6.18 -> 5.90 ms, with a barrier
// between the phases 5.78 (vortex 1.00 -> 0.91, 53,000 nodes 0.180 -> 0.170;
// blocks of 512 6.10, of 128 with barriers 6.07), and 5.88 with the threads
// that have no face meeting it too, as it has to be.
constexpr int kCharThreads = 256;
template <int MB>
__global__ void __launch_bounds__(kCharThreads, MB) k_face_char(LatView g, FaceScratch fs, int n1, int d0)
{
    const int n = fs.n0 + (blockIdx.x / 5u) * blockDim.x + threadIdx.x;
    ex::char_node(g, fs, n, d0 + blockIdx.y, blockIdx.x % 5u, n < n1, ex::BlockSync{});
}

// blocks of 256: TGV 128^3 2.00 -> 1.97 ms, vortex 64^3 0.338 -> 0.330 (128); 2.04 with 384
__global__ void __launch_bounds__(256, 3) k_face_back(LatView g, FaceScratch fs, int n1)
{
    const int n = fs.n0 + (blockIdx.x / 5u) * blockDim.x + threadIdx.x;
    if (n < n1) ex::back_node(g, fs, n, blockIdx.y, blockIdx.x % 5u);
}

__global__ void __launch_bounds__(128, 4) k_face_flux(LatView g, FaceScratch fs, int n1)
{
    const int n = fs.n0 + (blockIdx.x * blockDim.x + threadIdx.x) / 2;
    ex::flux_node(g, fs, n < n1 ? n : n1 - 1, blockIdx.y, n < n1);
}

void face_char(const LatView &g, const FaceScratch &fs, int n1, int mb, int d0, int nd, cudaStream_t st)
{
    const dim3 grid(5 * blocks_for(n1 - fs.n0, kCharThreads), nd);   // the five fields of 256 faces are neighbouring blocks
    if (mb == 2) k_face_char<2><<<grid, kCharThreads, 0, st>>>(g, fs, n1, d0);
    else if (mb == 3) k_face_char<3><<<grid, kCharThreads, 0, st>>>(g, fs, n1, d0);
    else k_face_char<4><<<grid, kCharThreads, 0, st>>>(g, fs, n1, d0);
}

}  // namespace

void fp64_geometry(const StructuredLaunch &S)
{
    const LatView g = make_view(S, 0.0, nullptr);
    fp64_geometry(g, S.kn, S.del, S.stream);
}

void fp64_geometry(const LatView &g, double *kn, double *del, cudaStream_t st)
{
    k_geometry<<<dim3(blocks_for(g.N, 128), kn ? 3 : 1), 128, 0, st>>>(g, kn, del);
}

int fp64_faces(const StructuredLaunch &S, const LatView &g, cudaStream_t st, const std::function<void(const char *)> &mark)
{
    int launches = 0;
    const bool one = g.N <= S.fs_ld;   // a single round: each kernel is its own timed entry
    for (int n0 = 0; n0 < g.N; n0 += S.fs_ld) {
        const FaceScratch fs{S.fs, n0, S.fs_ld};
        const int n1 = g.N - n0 < S.fs_ld ? g.N : n0 + S.fs_ld;
        const unsigned nb = blocks_for(n1 - n0, 128);
        k_face_base<<<dim3(nb, 3), 128, 0, st>>>(g, fs, n1);
        if (one) mark("face_base");
        const int *mb = S.face_mb;
        if (mb[0] == mb[1] && mb[0] == mb[2]) {
            face_char(g, fs, n1, mb[0], 0, 3, st);
            launches += 4;
        } else {
            for (int d = 0; d < 3; ++d) face_char(g, fs, n1, mb[d], d, 1, st);
            launches += 6;
        }
        if (one) mark("face_char");
        k_face_back<<<dim3(5 * blocks_for(n1 - n0, 256), 3), 256, 0, st>>>(g, fs, n1);
        if (one) mark("face_back");
        k_face_flux<<<dim3(blocks_for(2LL * (n1 - n0), 128), 3), 128, 0, st>>>(g, fs, n1);
        if (one) mark("face_flux");
    }
    if (!one) mark("faces");
    return launches;
}

}  // namespace cfd
