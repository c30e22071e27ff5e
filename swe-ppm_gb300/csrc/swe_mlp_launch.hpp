// Launchers of the surrogate's domain kernels (swe_mlp.cu), called by the
// domain entry points of swe_capi.cu.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "swe_device.cuh"

struct swe_mlp;

namespace swegb {
namespace mlp {

/// up to 128 consecutive edges of one column of one block: x-edges
/// (col | col+1) of rows j0 .. j0+count-1 (dir 0), or y-edges (j | j+1) of
/// column col for j = j0 .. j0+count-1 (dir 1).  Both sides of every edge are
/// contiguous in the column layout, so a tile's loads coalesce.  dir 2: the
/// y-edges (j0 | j0+1) of columns col .. col+count-1.
struct EdgeTile {
    int block, dir, col, j0, count;
};

/// net updates of every edge (hUpdL, hUpdR, huUpdL, huUpdR with the normal
/// momentum), stored at the element offset of the edge's left / lower cell
struct EdgeUpdates {
    float *x[4];
    float *y[4];
};

/// x-edges (0|1) .. (nx|nx+1) of rows 1..ny and y-edges (0|1) .. (ny|ny+1) of
/// columns 1..nx of every block: the edges one unsplit step solves
/// (src/blocks/SWE_DimensionalSplittingMpi.cpp:382-412), in tiles
inline std::vector<EdgeTile> buildEdgeTiles(const std::vector<BlockDesc> &blocks) {
    std::vector<EdgeTile> t;
    for (int k = 0; k < int(blocks.size()); k++) {
        const BlockDesc &B = blocks[k];
        for (int col = 0; col <= B.nx; col++)
            for (int j0 = 1; j0 <= B.ny; j0 += 128) t.push_back({k, 0, col, j0, std::min(128, B.ny - j0 + 1)});
        for (int col = 1; col <= B.nx; col++)
            for (int j0 = 0; j0 <= B.ny; j0 += 128) t.push_back({k, 1, col, j0, std::min(128, B.ny + 1 - j0)});
    }
    return t;
}

/// the same edges for the edge pass.  A column has ny+1 y-edges, so where ny is
/// a multiple of 128 its last tile would hold one edge: those blocks' lowest
/// y-edges (0|1) go to tiles along the row instead (512-row blocks: 8 tiles per
/// column instead of 9, the edge pass of the augmented solver at 2048^2 144 ->
/// 132 us).
///
/// The pass gives each of `ranges` workers a contiguous part of the list.  The
/// list is ordered so that each part holds pairs of tiles from all over the
/// domain, dealt out in turn (what is left of a full round split evenly): every
/// worker gets its share of the cheap (dry) parts, which as one stretch left
/// SMs idle at the end.  16 steps of the 4096^2 shoreline 11.20 -> 10.98 ms, 4
/// surrogate steps at 2048^2 2636 -> 2563 us, the augmented step at 1500^2 113 ->
/// 103 us; no size got slower, as 2048^2 in 512^2 blocks did by 4% with 8 tiles
/// in the place of a pair.
inline std::vector<EdgeTile> buildStepTiles(const std::vector<BlockDesc> &blocks, int ranges) {
    std::vector<EdgeTile> t;
    for (int k = 0; k < int(blocks.size()); k++) {
        const BlockDesc &B = blocks[k];
        const int first = B.ny % 128 == 0 ? 1 : 0;
        for (int col = 0; col <= B.nx; col++)
            for (int j0 = 1; j0 <= B.ny; j0 += 128) t.push_back({k, 0, col, j0, std::min(128, B.ny - j0 + 1)});
        for (int col = 1; col <= B.nx; col++)
            for (int j0 = first; j0 <= B.ny; j0 += 128) t.push_back({k, 1, col, j0, std::min(128, B.ny + 1 - j0)});
        for (int col = 1; first && col <= B.nx; col += 128) t.push_back({k, 2, col, 0, std::min(128, B.nx + 1 - col)});
    }
    if (ranges < 2) return t;
    constexpr int run = 2;
    const long long n = (long long)t.size(), full = n / (ranges * run) * run, left = n - full * ranges;
    if (!full) return t;
    std::vector<EdgeTile> p(t.size());
    size_t at = 0;
    for (long long w = 0; w < ranges; w++) {
        for (long long k = 0; k < full; k++) p[at++] = t[size_t((k / run * ranges + w) * run + k % run)];
        for (long long i = left * w / ranges; i < left * (w + 1) / ranges; i++) p[at++] = t[size_t(full * ranges + i)];
    }
    return p;
}

/// workers of the augmented solver's edge pass on the current device (all its
/// resident CTAs)
int edgeRanges();
/// the edge pass: every edge's net updates and the groups' max wave speed
/// (m null: the augmented Riemann solver on every edge, through the same
/// kernels); *used counts the edges the surrogate solved
cudaError_t launchSurrogateEdges(const DomainDev &d, const swe_mlp *m, const EdgeTile *tiles, int ntiles, EdgeUpdates u,
                                 unsigned long long *used, cudaStream_t s);
/// dt of every group from its max wave speed (unsplit step)
cudaError_t launchSurrogateDt(const DomainDev &d, int ngroups, cudaStream_t s);
/// the unsplit update of every interior cell from the stored net updates
cudaError_t launchSurrogateApply(const DomainDev &d, EdgeUpdates u, int nblocks, long long maxCells, cudaStream_t s);
/// time, step count and current buffer of every group
cudaError_t launchSurrogateFinish(const DomainDev &d, int ngroups, cudaStream_t s);
/// edge-state logger: slot e / stride of every stride-th edge gets the edge's
/// six inputs, its augmented-solver net updates and a wet flag (11 x nslots)
cudaError_t launchLogEdges(const DomainDev &d, const EdgeTile *tiles, int ntiles, int stride, float *slots,
                           long long nslots, cudaStream_t s);

/// SWE_GPU_ERR_DEVICE (message set) when a tensor-core wait of the surrogate
/// ran out of its iteration limit since the last check; waits for the device
int checkDeviceError(swe_mlp *m, const char *what);
/// the CUDA device the surrogate's state lives on
int deviceOf(const swe_mlp *m);

} // namespace mlp
} // namespace swegb
