// Step kernels instantiated for the augmented Riemann solver and the hybrid
// (f-wave / augmented) solver.
#include "swe_launch.hpp"
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
template <int S> static cudaError_t update(const DomainDev &d, int n, int th, cudaStream_t s) {
    return d.semantics == SEM_SPLIT
               ? launchPdlSmem(sweepKernel<S, SEM_SPLIT, true, false>, dim3(n), dim3(th), sizeof(SweepShared), s, d)
               : launchPdlSmem(sweepKernel<S, SEM_UNSPLIT, true, false>, dim3(n), dim3(th), sizeof(SweepShared), s, d);
}
template <int S> static cudaError_t lastEdge(const DomainDev &d, int ngroups, cudaStream_t s) {
    return launchPdl(lastEdgeKernel<S>, dim3((ngroups + 31) / 32), dim3(32), s, d, ngroups);
}

cudaError_t launchSpeedAug(const DomainDev &d, int n, int th, cudaStream_t s, bool pdl) {
    return d.solver == SOLVER_AUGRIE ? speed<SOLVER_AUGRIE>(d, n, th, s, pdl) : speed<SOLVER_HYBRID>(d, n, th, s, pdl);
}
cudaError_t launchLastEdgeAug(const DomainDev &d, int ngroups, cudaStream_t s) {
    return d.solver == SOLVER_AUGRIE ? lastEdge<SOLVER_AUGRIE>(d, ngroups, s) : lastEdge<SOLVER_HYBRID>(d, ngroups, s);
}
cudaError_t launchUpdateAug(const DomainDev &d, int n, int th, cudaStream_t s) {
    return d.solver == SOLVER_AUGRIE ? update<SOLVER_AUGRIE>(d, n, th, s) : update<SOLVER_HYBRID>(d, n, th, s);
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

int occupancyAug(int solver, int sem, bool update, int threads) {
    return solver == SOLVER_AUGRIE ? occupancy<SOLVER_AUGRIE>(sem, update, threads)
                                   : occupancy<SOLVER_HYBRID>(sem, update, threads);
}

} // namespace swegb
