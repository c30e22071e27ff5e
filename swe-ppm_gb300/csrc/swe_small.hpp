// Several time steps of a small domain in one cooperative launch
// (swe_small.cu), called by the domain entry points of swe_capi.cu.
#pragma once

#include <cuda_runtime.h>

#include "swe_device.cuh"

namespace swegb {
namespace small {

/// Meeting point of a dt group's CTAs, zero before the first launch; every
/// meeting leaves count at 0 and speed at 0.
struct __align__(128) Sync {
    unsigned count;            // CTAs that have arrived
    unsigned speed;            // the step's largest wave speed so far (float bits)
    unsigned long long epoch;  // (meetings so far << 32) | dt bits of the last one that formed a dt
    int ctas;                  // CTAs of the group
    int first;                 // the group's first CTA (publishes the clock)
};

constexpr int kMaxCols = 4;  // most columns of a CTA's segment
/// ... of a solver's.  The augmented one's edges bound a CTA, and at two columns
/// it lost to the passes when the line was drawn (400^2: 28 us a step against
/// 24); with its edges as they are now, two columns take 13.8 us there and the
/// passes 17.5
constexpr int maxCols(int solver) { return solver == SOLVER_AUGRIE ? 1 : kMaxCols; }

/// CTAs of `threads` rows and up to `cols` columns (1, 2 or 4, at most
/// maxCols(solver)) that are resident at once on the current device; 0 when it
/// cannot launch them together
int capacity(int solver, int cols, int threads);

/// Whether work on the stream can have the whole device, as capacity() takes it
/// to.  The SMs of a green context are a part of it, and a cooperative launch
/// that does not fit that part is not refused but never starts: such streams
/// (and any that cannot be told) take the passes, which need no CTAs together.
bool wholeDevice(cudaStream_t s);

/// Whether launch() failed because its CTAs cannot be resident together (a
/// context with fewer SMs than the device says): the passes run all the same
bool refused(cudaError_t e);

/// up to nsteps unsplit steps of every group that has not reached its target
/// (fewer once it has); units[i] is CTA i's segment of at most `cols` columns
cudaError_t launch(const DomainDev &d, const WorkUnit *units, int nunits, Sync *sync, int nsteps, int cols, int threads,
                   cudaStream_t s);

} // namespace small
} // namespace swegb
