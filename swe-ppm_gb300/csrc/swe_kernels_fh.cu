// Step kernels instantiated for the f-wave and HLLE solvers.
#include "swe_launch.hpp"
#include "swe_bound.cuh"
#include "swe_sweep.cuh"

namespace swegb {

template <int S> static cudaError_t speed(const DomainDev &d, int n, int th, cudaStream_t s, bool pdl) {
    if (d.semantics == SEM_SPLIT) {
        if (pdl) return launchPdl(speedSplitKernel<S>, dim3(n), dim3(th), s, d);
        speedSplitKernel<S><<<n, th, 0, s>>>(d);
        return cudaGetLastError();
    }
    if (pdl) return launchPdlSmem(sweepKernel<S, SEM_UNSPLIT, false, false>, dim3(n), dim3(th), sizeof(SweepShared), s, d);
    sweepKernel<S, SEM_UNSPLIT, false, false><<<n, th, sizeof(SweepShared), s>>>(d);
    return cudaGetLastError();
}
template <int S> static cudaError_t update(const DomainDev &d, int n, int th, int groups, cudaStream_t s) {
    if (groups == kTeamGroups && d.semantics == SEM_UNSPLIT) {
        const auto k = sweepKernel<S, SEM_UNSPLIT, true, true>;
        constexpr int smem = kTeamGroups * int(sizeof(SweepShared));
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        return launchPdlSmem(k, dim3(n / kTeamGroups), dim3(th * kTeamGroups), smem, s, d);
    }
    return d.semantics == SEM_SPLIT
               ? launchPdlSmem(sweepKernel<S, SEM_SPLIT, true, false>, dim3(n), dim3(th), sizeof(SweepShared), s, d)
               : launchPdlSmem(sweepKernel<S, SEM_UNSPLIT, true, false>, dim3(n), dim3(th), sizeof(SweepShared), s, d);
}
template <int S> static cudaError_t lastEdge(const DomainDev &d, int ngroups, cudaStream_t s) {
    return launchPdl(lastEdgeKernel<S>, dim3((ngroups + 31) / 32), dim3(32), s, d, ngroups);
}

cudaError_t launchSpeedFH(const DomainDev &d, int n, int th, cudaStream_t s, bool pdl) {
    return d.solver == SOLVER_FWAVE ? speed<SOLVER_FWAVE>(d, n, th, s, pdl) : speed<SOLVER_HLLE>(d, n, th, s, pdl);
}
cudaError_t launchLastEdgeFH(const DomainDev &d, int ngroups, cudaStream_t s) {
    return d.solver == SOLVER_FWAVE ? lastEdge<SOLVER_FWAVE>(d, ngroups, s) : lastEdge<SOLVER_HLLE>(d, ngroups, s);
}
cudaError_t launchUpdateFH(const DomainDev &d, int n, int th, int groups, cudaStream_t s) {
    return d.solver == SOLVER_FWAVE ? update<SOLVER_FWAVE>(d, n, th, groups, s) : update<SOLVER_HLLE>(d, n, th, groups, s);
}

cudaError_t launchSpeedBound(const DomainDev &d, int grid, cudaStream_t s) {
    cudaError_t e = d.solver == SOLVER_FWAVE ? launchPdl(speedBoundKernel<SOLVER_FWAVE>, dim3(grid), dim3(256), s, d)
                                             : launchPdl(speedBoundKernel<SOLVER_HLLE>, dim3(grid), dim3(256), s, d);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

template <class K> static int occ(K kernel, int th, size_t smem = 0) {
    int a = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, kernel, th, smem);
    return a;
}

/// resident CTAs per SM of one pass's kernel
template <int S> static int occupancy(int sem, bool upd, int th) {
    const bool split = sem == SEM_SPLIT;
    return upd ? (split ? occ(sweepKernel<S, SEM_SPLIT, true, false>, th, sizeof(SweepShared))
                        : occ(sweepKernel<S, SEM_UNSPLIT, true, false>, th, sizeof(SweepShared)))
               : (split ? occ(speedSplitKernel<S>, th) : occ(sweepKernel<S, SEM_UNSPLIT, false, false>, th, sizeof(SweepShared)));
}

int occupancyFH(int solver, int sem, bool update, int threads) {
    return solver == SOLVER_FWAVE ? occupancy<SOLVER_FWAVE>(sem, update, threads)
                                  : occupancy<SOLVER_HLLE>(sem, update, threads);
}

int occupancyBound(int solver) {
    return solver == SOLVER_FWAVE ? occ(speedBoundKernel<SOLVER_FWAVE>, 256) : occ(speedBoundKernel<SOLVER_HLLE>, 256);
}

} // namespace swegb
