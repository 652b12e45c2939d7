// static_stage.cu -- one SSP-RK3 stage on a periodic lattice that allocates
// no device memory.
//
// Some callers cannot call cudaMalloc while they advance a solution: code
// that runs inside a host framework owning a fixed device-memory pool, a
// real-time loop where an allocation (and the implicit device synchronisation
// that cudaMalloc/cudaFree may cause) is not allowed, or a plugin that is only
// handed buffers.  For them, cfd_lattice_stage_static runs the same kernels
// as the resident solver's structured path, but keeps every intermediate of
// the stage (structure-of-arrays copies of the inputs, node fluxes, viscous
// fluxes, face fluxes, the error word) in one library-owned array declared
// below, sized for at most CFD_STATIC_MAX_NODES lattice nodes.
//
// The array exists once per GPU that loads the library and stays allocated
// until the process exits.  All calls share it: two calls whose work
// overlaps on the GPU (different streams, or different host threads using
// the same device) race on it and produce garbage; callers must serialise
// them.  Host code cannot use the array's name as a device address, so the
// first call on each device looks the address up with cudaGetSymbolAddress
// (with that device current) and caches it; make that first call before any
// stream capture begins.  The cached address belongs to the device's
// current context: after cudaDeviceReset the process must not call the
// entry point again.
#include <mutex>

#include "internal.h"
#include "structured.h"

namespace cfd {
namespace {

// doubles per lattice node held in the scratch array:
//   geometry SoA 22 (9 node metrics, det, 3x3 face metrics, 3 face dets),
//   FLOW 9, U0/U1/U2 15, Q 5, node fluxes 15, viscous fluxes 15,
//   sqrt(rho) and its products with u, v, w, H 5, unit normals 9, filter
//   width 1, hand-over between the face kernels 126, face fluxes 15, L 5
constexpr size_t kPerNode = 22 + 9 + 15 + 5 + 15 + 15 + 5 + 9 + 1 + 3 * kFaceScratch + 15 + 5;   // 242
constexpr size_t kFlagDoubles = 32;                                    // 256 B for the error word
constexpr size_t kScratchDoubles = (size_t)CFD_STATIC_MAX_NODES * kPerNode + kFlagDoubles;
static_assert(kScratchDoubles * 8 / 1000000 == 63, "cfd_rhs.h states the size");

static __device__ __align__(256) double g_stage_scratch[kScratchDoubles];

constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
double *g_scratch_addr[kMaxDevices] = {};

// Device address of the scratch array on the current device (looked up once
// per device).
cfd_status_t scratch_address(double **out)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return CFD_ECUDA;
    if (dev < 0 || dev >= kMaxDevices) return CFD_EUNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_addr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_stage_scratch);
        if (e != cudaSuccess || !p) return CFD_ECUDA;
        g_scratch_addr[dev] = (double *)p;
    }
    *out = g_scratch_addr[dev];
    return CFD_OK;
}

// The stage's inputs and results in the reference layout, rows 1..N.
struct Rows {
    const double *det, *deter, *metric;
    double *U[3], *flow, *L;
};

// Reference rows -> SoA in one launch, a thread per node and component, and
// the error word to zero.  Components of a node, in the order of the scratch
// array's first 46 rows: det after the 9 node metrics, the 3x3 face
// metrics, 3 face dets, FLOW, U0, U1, U2.  On a few thousand nodes a launch
// costs 3 us whatever it moves: twelve of them, a memset and four for the
// results were 55 of the 222 us of a stage on 17^3 nodes.
constexpr int kIn = 46;
__global__ void __launch_bounds__(256) k_rows_to_soa(Rows R, long long N, double *__restrict__ soa, unsigned *flags)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) *flags = 0;
    if (t >= N * kIn) return;
    const long long n = t / kIn, r = n + 1;
    const int c = (int)(t % kIn);
    double v;
    if (c < 9) v = R.metric[r * 63 + c];
    else if (c == 9) v = R.det[r];
    else if (c < 19) {
        const int d = (c - 10) / 3;
        v = R.metric[r * 63 + 9 * (1 + 2 * d) + (c - 10)];   // row d of the face metric of face d
    } else if (c < 22) v = R.deter[r * 6 + 2 * (c - 19)];
    else if (c < 31) v = R.flow[r * 9 + (c - 22)];
    else {
        const int q = (c - 31) / 5;
        v = R.U[q][r * 5 + (c - 31) % 5];
    }
    soa[c * N + n] = v;
}

// Results back into the caller's rows: FLOW, U_j (U_Q's output), the U the
// stage advanced, and L.
__global__ void __launch_bounds__(256)
k_soa_to_rows(Rows R, long long N, const double *__restrict__ flow, const double *__restrict__ Uj, int j,
              const double *__restrict__ Ua, int advanced, const double *__restrict__ L)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * 9) return;
    const long long n = t / 9, r = n + 1;
    const int c = (int)(t % 9);
    R.flow[r * 9 + c] = flow[c * N + n];
    if (c >= 5) return;
    R.U[j][r * 5 + c] = Uj[c * N + n];
    R.U[advanced][r * 5 + c] = Ua[c * N + n];
    if (R.L) R.L[r * 5 + c] = L[c * N + n];
}

}  // namespace
}  // namespace cfd

extern "C" cfd_status_t cfd_lattice_stage_static(void *cuda_stream, int32_t ni, int32_t nj, int32_t nk, int32_t j,
                                                 double del_t, const cfd_params_t *params, const double *det,
                                                 const cfd_determ_t *deter, const cfd_metric_t *metric,
                                                 cfd_column_t *U0, cfd_column_t *U1, cfd_column_t *U2,
                                                 cfd_flow_t *FLOW, cfd_column_t *L_out)
{
    using namespace cfd;
    if (ni < 1 || nj < 1 || nk < 1 || j < 0 || j > 2) return CFD_EINVAL;
    const long long N = (long long)ni * nj * nk;
    if (N > CFD_STATIC_MAX_NODES) return CFD_EINVAL;   // beyond the static scratch array
    if (!det || !deter || !metric || !U0 || !U1 || !U2 || !FLOW) return CFD_EINVAL;
    if (params && params->precision != CFD_PREC_FP64) return CFD_EUNSUPPORTED;   // FP64 form only
    if (cudaPeekAtLastError() != cudaSuccess) return CFD_ECUDA;   // an earlier error, left for the caller
    double *base = nullptr;
    cfd_status_t s = scratch_address(&base);
    if (s != CFD_OK) return s;
    cudaStream_t st = (cudaStream_t)cuda_stream;

    // carve the scratch array (N nodes used, SoA [component][N])
    double *p = base;
    auto take = [&](size_t comps) {
        double *q = p;
        p += comps * (size_t)N;
        return q;
    };
    StructuredLaunch S{};
    S.ni = ni;
    S.nj = nj;
    S.nk = nk;
    S.stream = st;
    S.P = make_phys(params);
    S.mixed = 0;
    S.m9 = take(9);   // the inputs, in k_rows_to_soa's order
    S.det = take(1);
    S.fm = take(9);
    S.fdet = take(3);
    S.prim9 = take(9);
    S.U[0] = take(5);
    S.U[1] = take(5);
    S.U[2] = take(5);
    S.Q = take(5);
    S.FEG = take(15);
    S.V = take(15);
    S.sh = take(5);
    S.kn = take(9);
    S.del = take(1);
    S.fs = take(3 * kFaceScratch);
    S.fs_ld = (int)N;
    S.Fh = take(15);
    double *Lsoa = take(5);
    S.flags = (unsigned *)(base + (size_t)CFD_STATIC_MAX_NODES * kPerNode);

    // every region is written before it is read within this call
    const Rows R{det, (const double *)deter, (const double *)metric,
                 {(double *)U0, (double *)U1, (double *)U2}, (double *)FLOW, (double *)L_out};
    k_rows_to_soa<<<blocks_for(N * kIn, 256), 256, 0, st>>>(R, N, base, S.flags);

    fp64_geometry(S);
    structured_stage(S, j, del_t, L_out ? Lsoa : nullptr);

    const int advanced = j == 0 ? 1 : (j == 1 ? 2 : 0);
    k_soa_to_rows<<<blocks_for(N * 9, 256), 256, 0, st>>>(R, N, S.prim9, S.U[j], j, S.U[advanced], advanced, Lsoa);

    // peek, not get: a failed launch stays readable by the caller's own checks
    cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) return CFD_ECUDA;
    unsigned flags = 0;
    e = cudaMemcpyAsync(&flags, S.flags, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return CFD_ECUDA;
    if (flags & CFD_FLAG_NONFINITE) return CFD_ENONFINITE;
    return CFD_OK;
}
