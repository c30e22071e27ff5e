// The unsplit step of a small domain (exact arithmetic), several steps in one
// cooperative launch.
//
// A 256^2 step is two launches of a few microseconds of work each, and spent
// its time on launch latency, on the descriptor and state loads at the start
// of each, and on solving every edge twice.  Here one CTA keeps its segment (up
// to 256 rows x up to 4 columns, a row per thread) in registers over all steps
// and solves each edge once:
//   - cells across the segment's sides come from the current buffer (through
//     L2: other CTAs wrote them), the rest from registers and shared memory;
//   - the edges' net updates are summed per cell in the order of the update
//     pass (sweepKernel), their speeds reduced over the group's CTAs;
//   - the group meets; the last CTA turns the speed into maxTimestep
//     (src/blocks/SWE_DimensionalSplittingMpi.cpp:448-456) and publishes it
//     with the meeting's number in one word, so that who waits needs no second
//     load;
//   - the update with the dry clamp (:484-518), the ghost pushes of the block's
//     rim, and a second meeting before the next step reads the new cells.
// Every wait is bounded; a CTA whose wait runs out leaves (giveUp), and no later
// launch steps the group again.
//
// Bound by the two meetings (about 1.5 us each) and the edges' latency, not by
// bandwidth or issue.  256^2 hybrid step: 12.3 us as two passes, 7.2 us here.
#include <cudaTypedefs.h>

#include "swe_small.hpp"
#include "swe_sweep.cuh"

namespace swegb {
namespace small {

constexpr unsigned kSpinLimit = 1u << 22;

/// waits (bounded) until the group's meeting after number `seen` is over:
/// its epoch word, or `seen` unchanged in the upper half when the limit ran out
__device__ __forceinline__ unsigned long long awaitEpoch(Sync *y, unsigned seen) {
    unsigned long long e = 0;
    for (unsigned n = 0; n < kSpinLimit; ++n) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(e) : "l"(&y->epoch) : "memory");
        if (unsigned(e >> 32) != seen) return e;
    }
    return (unsigned long long)seen << 32;
}
__device__ __forceinline__ void publishEpoch(Sync *y, unsigned number, float dt) {
    const unsigned long long e = (unsigned long long)number << 32 | __float_as_uint(dt);
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(&y->epoch), "l"(e) : "memory");
}

/// A CTA leaves without its meeting: status bit 3, and for a caller who reads no
/// status (the allocation-free call has none) dt and the depths that this CTA
/// was to write are NaN.
static __device__ __noinline__ void giveUp(GroupState *G, float *H, unsigned pitch, int columns) {
    if (threadIdx.x == 0) {
        atomicOr(&G->status, 8);
        atomicExch(&G->dt, NAN);
    }
    for (int c = 0; c < columns; c++) H[size_t(c) * pitch] = NAN;
}

template <int S, int XC>
__global__ void __launch_bounds__(kMaxTileRows, XC > 2 ? 3 : 4)
    smallStepKernel(const DomainDev d, const WorkUnit *units, Sync *sync, int nsteps) {
    __shared__ float sC[2][6][kMaxTileRows];  // y-direction cell quantities of a column
    __shared__ float sR[2][2][kMaxTileRows];  // right-going (h, hv) update into row t
    __shared__ float sHalo[2][6][XC];         // cells below / above the segment
    __shared__ float sRed[kMaxTileRows / 32];
    __shared__ float sDt;
    __shared__ int sGo;
    __shared__ int sDead;           // an earlier meeting ran out: the meeting point is not to be used
    __shared__ unsigned sDtBefore;  // the dt that the leader replaces at the end

    const int t = threadIdx.x, TY = blockDim.x;
    const WorkUnit wu = units[blockIdx.x];
    const BlockDesc B = d.blocks[wu.block];
    const int nx = B.nx, ny = B.ny;
    const long long base = B.base;
    const float dx = B.dx, dy = B.dy;
    GroupState *G = d.groups + B.group;
    if (!groupActive(G)) return;  // the whole group alike
    Sync *Y = sync + B.group;
    int cur = G->cur;
    float time = G->time;
    const float target = G->target;
    const int need = Y->ctas;
    if (t == 0) {  // (thread 0's alone, here to leave the registers to the edges)
        sDead = G->status & 8;
        sDtBefore = __float_as_uint(G->dt);
    }
    const bool leader = Y->first == int(blockIdx.x);
    // the meetings' number before this launch's first one: it cannot move
    // before every CTA of the group, this one included, has arrived
    unsigned seen = unsigned(*(volatile unsigned long long *)&Y->epoch >> 32);

    const int n = wu.x1 - wu.x0, x0 = wu.x0, y0 = wu.y0, y = y0 + t;
    const int yTop = min(y0 + TY - 1, ny), last = yTop - y0;
    const bool active = t <= last;
    const unsigned P = unsigned(B.pitch);
    const float *BT = d.b + base;

    // a rim row's ghost: one store per field at rimGhost + x * rimPitch, as in
    // the update pass (0: none, 1: copy, 2: copy with -hv, 3: keep); the first
    // and last column's inline too.  (All through pushGhosts: 256^2 hybrid 7.36
    // us a step, 7.07 so; with the descriptor by reference instead of copied a
    // single step is 5% slower.)
    const bool rimRow = active && (y == 1 || y == ny);
    int rimMode = 0, rimPitch = int(P);
    long long rimGhost = 0;
    if (rimRow && ny > 1) {
        const int side = (y == 1) ? 2 : 3, type = B.bnd[side];
        rimGhost = (side == 2) ? 0 : ny + 1;
        rimMode = 3;
        if (type == OUTFLOW || type == WALL) {
            rimMode = type == WALL ? 2 : 1;
        } else if (type == CONNECT_WITHIN_RANK) {
            const BlockDesc &N = d.blocks[B.nbr[side]];
            rimMode = 1;
            rimGhost = N.base - base + ((side == 2) ? N.ny + 1 : 0);
            rimPitch = N.pitch;
        }
    }

    float qh[XC], qhu[XC], qhv[XC], qb[XC];
#pragma unroll
    for (int c = 0; c < XC; c++) {
        qh[c] = 1.f;
        qhu[c] = qhv[c] = qb[c] = 0.f;
        if (c < n && active) {
            const unsigned o = unsigned(x0 + c) * P + unsigned(y);
            qh[c] = __ldcg(pick(d.h, cur) + base + o);
            qhu[c] = __ldcg(pick(d.hu, cur) + base + o);
            qhv[c] = __ldcg(pick(d.hv, cur) + base + o);
            qb[c] = __ldg(BT + o);
        }
    }
    float dt = 0.f;
    bool bad = false;
    int done = 0;
    while (done < nsteps && time < target) {
        const float *H = pick(d.h, cur) + base, *HU = pick(d.hu, cur) + base, *HV = pick(d.hv, cur) + base;
        // the cells across the segment's sides: left and right column of this
        // row, and (threads 0 .. 2n-1) one cell below or above
        float lh = 1.f, lhu = 0.f, lhv = 0.f, lb = 0.f, rh = 1.f, rhu = 0.f, rhv = 0.f, rb = 0.f;
        if (active) {
            const unsigned o = unsigned(x0 - 1) * P + unsigned(y), p = unsigned(x0 + n) * P + unsigned(y);
            lh = __ldcg(H + o); lhu = __ldcg(HU + o); lhv = __ldcg(HV + o); lb = __ldg(BT + o);
            rh = __ldcg(H + p); rhu = __ldcg(HU + p); rhv = __ldcg(HV + p); rb = __ldg(BT + p);
        }
        for (int i = t; i < 2 * n; i += TY) {
            const int up = i >= n ? 1 : 0, c = i - up * n;
            const unsigned o = unsigned(x0 + c) * P + unsigned(up ? yTop + 1 : y0 - 1);
            Cell dummy, q;
            cellQuantities<S>(__ldcg(H + o), 0.f, __ldcg(HV + o), __ldg(BT + o), dummy, q);
            sHalo[up][0][c] = q.h; sHalo[up][1][c] = q.hn; sHalo[up][2][c] = q.b;
            sHalo[up][3][c] = q.u; sHalo[up][4][c] = q.sq; sHalo[up][5][c] = q.c;
        }
        float smax = 0.f, sxH[XC], sxHU[XC], syH[XC], syHV[XC], pendH = 0.f, pendHU = 0.f;
        Cell prevX, unused;
        cellQuantities<S>(lh, lhu, lhv, lb, prevX, unused);
#pragma unroll
        for (int c = 0; c <= XC; c++) {
            if (c > n) break;
            const bool own = c < XC && c < n;
            const int k = c < XC ? c : 0;
            Cell cx, cy;
            cellQuantities<S>(own ? qh[k] : rh, own ? qhu[k] : rhu, own ? qhv[k] : rhv, own ? qb[k] : rb, cx, cy);
            if (active) {  // x-edge (x0+c-1 | x0+c)
                float aL, aR, auL, auR, s;
                edgeSolve<S, true>(prevX, cx, aL, aR, auL, auR, s);
                smax = vmax(smax, s);
                if (c > 0) {
                    sxH[c > 0 ? c - 1 : 0] = pendH + aL;
                    sxHU[c > 0 ? c - 1 : 0] = pendHU + auL;
                }
                pendH = aR;
                pendHU = auR;
            }
            prevX = cx;
            if (!own) break;
            // y-edges of column x0+c
            const int buf = c & 1;
            sC[buf][0][t] = cy.h; sC[buf][1][t] = cy.hn; sC[buf][2][t] = cy.b;
            sC[buf][3][t] = cy.u; sC[buf][4][t] = cy.sq; sC[buf][5][t] = cy.c;
            __syncthreads();
            float bLh = 0.f, bLhv = 0.f, rH = 0.f, rHV = 0.f;
            if (active) {
                const bool top = t == last;
                const float *q = top ? &sHalo[1][0][c] : &sC[buf][0][t + 1];
                const int w = top ? XC : kMaxTileRows;
                const Cell up = makeCell(q[0], q[w], q[2 * w], q[3 * w], q[4 * w], q[5 * w]);
                float bR, bRhv, s;
                edgeSolve<S, true>(cy, up, bLh, bR, bLhv, bRhv, s);
                smax = vmax(smax, s);
                if (!top) {
                    sR[buf][0][t + 1] = bR;
                    sR[buf][1][t + 1] = bRhv;
                }
                if (t == 0) {
                    const Cell low = makeCell(sHalo[0][0][c], sHalo[0][1][c], sHalo[0][2][c], sHalo[0][3][c],
                                              sHalo[0][4][c], sHalo[0][5][c]);
                    float a, av;
                    edgeSolve<S, true>(low, cy, a, rH, av, rHV, s);
                    smax = vmax(smax, s);
                }
            }
            __syncthreads();
            if (t > 0) {
                rH = sR[buf][0][t];
                rHV = sR[buf][1][t];
            }
            syH[k] = rH + bLh;
            syHV[k] = rHV + bLhv;
        }
        // the group's maximum speed, dt
        const float m = blockReduceMax(smax, sRed);
        if (t == 0) {
            if (!sDead) atomicMax(&Y->speed, __float_as_uint(m));
            if (sDead) {
                sGo = 0;
            } else if (arriveAcqRel(&Y->count, 1u) + 1u == unsigned(need)) {
                const float s = __uint_as_float(__ldcg(&Y->speed));
                const BlockDesc &F = d.blocks[G->firstBlock];
                dt = timestepFromSpeed(s, F.dx, F.dy, SEM_UNSPLIT);
                if (!(s == s)) atomicOr(&G->status, 1);
                G->speed = s;
                Y->speed = 0u;
                Y->count = 0u;
                publishEpoch(Y, seen + 1u, dt);
                sGo = 1;
            } else {
                const unsigned long long e = awaitEpoch(Y, seen);
                dt = __uint_as_float(unsigned(e));
                sGo = unsigned(e >> 32) != seen;
            }
            sDt = dt;
        }
        __syncthreads();
        seen++;
        if (!sGo) {
            giveUp(G, pick(d.h, cur ^ 1) + base + size_t(x0) * P + y, P, active ? n : 0);
            return;
        }
        dt = sDt;
        // Q^{n+1}, as the update pass forms it
        const float dtdx = dt / dx, dtdy = dt / dy;
        float *HO = pick(d.h, cur ^ 1) + base, *HUO = pick(d.hu, cur ^ 1) + base, *HVO = pick(d.hv, cur ^ 1) + base;
#pragma unroll
        for (int c = 0; c < XC; c++) {
            if (c >= n || !active) break;
            float hn = qh[c] - (dtdx * sxH[c] + dtdy * syH[c]);
            float hun = qhu[c] - dtdx * sxHU[c];
            float hvn = qhv[c] - dtdy * syHV[c];
            if (hn < 0.f) {
                hn = 0.f; hun = 0.f; hvn = 0.f;
            } else if (hn < 0.1f) {
                hun = 0.f; hvn = 0.f;
            }
            bad |= !(fabsf(hn) <= FLT_MAX);
            const int x = x0 + c;
            const unsigned o = unsigned(x) * P + unsigned(y);
            HO[o] = hn;
            HUO[o] = hun;
            HVO[o] = hvn;
            if (x == 1 || x == nx || rimRow) {
                bool call = rimRow && rimMode == 0;
                if (x == 1 || x == nx) {
                    const int side = x == 1 ? 0 : 1, type = B.bnd[side];
                    call = call || nx == 1 || ny == 1 || (type != OUTFLOW && type != WALL && type != CONNECT_WITHIN_RANK);
                    if (!call) {
                        const long long own = side ? (long long)(nx + 1) * P : 0;
                        long long g = own;
                        if (type == CONNECT_WITHIN_RANK) {
                            const BlockDesc &N = d.blocks[B.nbr[side]];
                            g = N.base - base + (side ? 0 : (long long)(N.nx + 1) * N.pitch);
                        }
                        HO[g + y] = hn;
                        HUO[g + y] = type == WALL ? -hun : hun;
                        HVO[g + y] = hvn;
                        if (rimRow) {  // the corner
                            const long long k = own + (y == 1 ? 0 : ny + 1);
                            HO[k] = hn;
                            HUO[k] = hun;
                            HVO[k] = hvn;
                        }
                    }
                }
                if (call) {
                    pushGhosts(d, B, cur ^ 1, P, x, y, hn, hun, hvn);
                } else if (rimRow) {
                    const long long g = rimGhost + (long long)x * rimPitch;
                    if (rimMode == 3) {
                        HO[g] = __ldcg(H + g);
                        HUO[g] = __ldcg(HU + g);
                        HVO[g] = __ldcg(HV + g);
                    } else {
                        HO[g] = hn;
                        HUO[g] = hun;
                        HVO[g] = rimMode == 2 ? -hvn : hvn;
                    }
                }
            }
            qh[c] = hn;
            qhu[c] = hun;
            qhv[c] = hvn;
        }
        time = time + dt;
        cur ^= 1;
        done++;
        if (done < nsteps && time < target) {  // the new cells are there before anyone reads them
            __syncthreads();
            if (t == 0) {
                if (arriveAcqRel(&Y->count, 1u) + 1u == unsigned(need)) {
                    Y->count = 0u;
                    publishEpoch(Y, seen + 1u, dt);
                    sGo = 1;
                } else {
                    sGo = unsigned(awaitEpoch(Y, seen) >> 32) != seen;
                }
            }
            __syncthreads();
            seen++;
            if (!sGo) {
                giveUp(G, pick(d.h, cur) + base + size_t(x0) * P + y, P, active ? n : 0);
                return;
            }
        }
    }
    if (__syncthreads_or(bad) && t == 0) atomicOr(&G->status, 2);
    if (leader && t == 0) {  // (every CTA of the group has read the state above before the first meeting)
        // (dt stays NaN where a CTA of the group has given up)
        atomicCAS(reinterpret_cast<unsigned *>(&G->dt), sDtBefore, __float_as_uint(dt));
        G->time = time;
        G->steps += done;
        G->cur = cur;
        G->ghostsAhead = 1;
        G->boundsValid[0] = 0;
        G->boundsValid[1] = 0;
        G->lastCandidates = G->tiles;  // every edge was evaluated
    }
}

namespace {

using Kernel = void (*)(const DomainDev, const WorkUnit *, Sync *, int);

template <int S> Kernel pickCols(int cols) {
    return cols == 1 ? smallStepKernel<S, 1> : cols == 2 ? smallStepKernel<S, 2> : smallStepKernel<S, kMaxCols>;
}
Kernel pickKernel(int solver, int cols) {
    switch (solver) {
    case SOLVER_FWAVE: return pickCols<SOLVER_FWAVE>(cols);
    case SOLVER_AUGRIE: return smallStepKernel<SOLVER_AUGRIE, 1>;  // (maxCols)
    case SOLVER_HYBRID: return pickCols<SOLVER_HYBRID>(cols);
    default: return pickCols<SOLVER_HLLE>(cols);
    }
}

} // namespace

int capacity(int solver, int cols, int threads) {
    int dev = 0, coop = 0, sms = 0, occ = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, pickKernel(solver, cols), threads, 0);
    return coop ? sms * occ : 0;
}

bool wholeDevice(cudaStream_t s) {
    // (looked up once; a driver without it has no green contexts)
    static const PFN_cuStreamGetGreenCtx_v12040 ask = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuStreamGetGreenCtx", &f, 12040, cudaEnableDefault, &q);
        if (e != cudaSuccess) cudaGetLastError();
        return reinterpret_cast<PFN_cuStreamGetGreenCtx_v12040>(e == cudaSuccess && q == cudaDriverEntryPointSuccess ? f : nullptr);
    }();
    CUgreenCtx green = nullptr;
    return !ask || (ask(s, &green) == CUDA_SUCCESS && !green);
}

bool refused(cudaError_t e) {
    return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported;
}

cudaError_t launch(const DomainDev &d, const WorkUnit *units, int nunits, Sync *sync, int nsteps, int cols, int threads,
                   cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(nunits));
    cfg.blockDim = dim3(unsigned(threads));
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, pickKernel(d.solver, cols), d, units, sync, nsteps);
    const cudaError_t last = cudaGetLastError();  // (clears a refusal's)
    return e != cudaSuccess ? e : last;
}

} // namespace small
} // namespace swegb
