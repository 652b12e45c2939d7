// rounds.h -- scratch of the face passes that run in rounds of rows or nodes:
// what a round takes is a matter of speed alone, so it gives way to the
// memory there is.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>

namespace cfd {

// Device memory for bytes(round) bytes: `round` halves, down to `least`,
// while that is more than half of what is free (the rest of the program
// allocates too) or cannot be had.  The rounds of a face pass hand nothing
// on, so any size gives the same bits; smaller ones cost launches (TGV
// 128^3 in rounds of 2^21, 2^19, 2^17 nodes: 37.7, 38.0, 39.3 ms; Weno case
// on 96^3 rows in rounds of 2^18, 2^16, 2^14: 18.2, 19.1, 23.3 ms).
template <class Bytes>
cudaError_t round_alloc(long long &round, long long least, const Bytes &bytes, void **p)
{
    for (;; round = std::max(least, (round + 1) / 2)) {
        size_t free_bytes = 0, total = 0;
        cudaError_t e = cudaMemGetInfo(&free_bytes, &total);
        if (e != cudaSuccess) return e;
        if (round > least && bytes(round) > free_bytes / 2) continue;
        e = cudaMalloc(p, bytes(round));
        if (e == cudaSuccess) return e;
        cudaGetLastError();
        if (e != cudaErrorMemoryAllocation || round <= least) return e;
    }
}
constexpr long long kLeastRound = 4096;   // rows or nodes of a round at least (or all of them): 4 to 5 MB

// Scratch of launch_uq and launch_weno for `rows` rows: the +1/2 faces
// [3][5][rows] and the -1/2 faces [3][5][rows] (doubles), then generation
// stamps [3][rows] (unsigned, zero when allocated); and the face kernels' own
// scratch for one round of rows, [3][kRowFace][round].
constexpr int kRowFace = 48;               // doubles of one row's face along one direction
constexpr long long kRowRound = 1 << 18;   // rows of a round at most: 302 MB, some 25 waves of blocks
static_assert(3 * kRowFace * 8 == 1152, "cfd_rhs.h states the bytes per row of a round");
struct RowScratch {
    double *face = nullptr;   // null: none, each row evaluates both faces itself
    double *col = nullptr;
    long long rows = 0, round = 0;
    unsigned *stamps() const { return reinterpret_cast<unsigned *>(face + 30 * rows); }
    bool serves(int n) const { return face && rows >= n; }
};
inline size_t row_face_bytes(long long rows) { return (size_t)rows * (30 * sizeof(double) + 3 * sizeof(unsigned)); }
inline size_t row_round_bytes(long long round) { return (size_t)round * 3 * kRowFace * sizeof(double); }
// Allocates it for `rows` rows on the current device, in rounds that leave
// half of the free memory (round_alloc).  On failure S stays empty.
cudaError_t row_scratch_alloc(RowScratch &S, long long rows);
void row_scratch_free(RowScratch &S);

}  // namespace cfd
