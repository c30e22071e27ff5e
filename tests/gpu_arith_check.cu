// Checks the edge arithmetic's known-range operators and the solvers' paths
// for tame operands against the general ones, bit for bit, on the device.
// Prints one line "name mismatches samples" per check.
#include <cstdio>
#include <cstdint>
#include <cuda_runtime.h>

#include "swe_device.cuh"
#include "swe_sweep.cuh"

using namespace swegb;

enum { RCP, SQRT, DIV, DIV_NEAR, FWAVE, HLLE, AUG, TAKEN, NCHECK };

__device__ uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__device__ bool count(unsigned long long *c, int k, bool bad) {
    if (bad) atomicAdd(c + k, 1ull);
    return bad;
}

/// every float of [2^-64, 2^64)
__global__ void unary(unsigned long long *c) {
    const uint32_t lo = (127u - 64u) << 23, n = 128u << 23;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float x = __uint_as_float(lo + i);
        count(c, RCP, !same(rcpRn(x), 1.f / x) || !same(rcpRn(-x), 1.f / -x));
        count(c, SQRT, !same(sqrtRn(x), sqrtf(x)));
    }
}

/// quotients: random ones, and ones next to the middle of two floats
__global__ void quotients(unsigned long long *c, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t z = mix(i), w = mix(z);
        const float b = __uint_as_float(uint32_t(w & 1) << 31 | uint32_t(127 - 60 + (w >> 8) % 120) << 23 | uint32_t(z & 0x7fffff));
        const float a = __uint_as_float(uint32_t(w >> 1 & 1) << 31 | uint32_t(127 - 60 + (w >> 24) % 120) << 23 | uint32_t(z >> 23 & 0x7fffff));
        count(c, DIV, !same(divRn(a, b), a / b));
        const float q = __uint_as_float(127u << 23 | uint32_t(z >> 23 & 0x7fffff));
        const float p = __uint_as_float(127u << 23 | uint32_t(z & 0x7fffff));
        const float m = float(double(p) * (double(q) + 0x1p-24));
        for (int k = -1; k <= 1; k++) {
            const float x = __uint_as_float(__float_as_uint(m) + k);
            count(c, DIV_NEAR, !same(divRn(x, p), x / p));
        }
    }
}

/// an edge from the hash: depths, momenta and beds of every size, zeros of
/// both signs, near-equal sides, shorelines, and now and then infinities and NaN
__device__ void randomEdge(uint64_t i, float e[6]) {
    uint64_t z = mix(i * 2 + 1);
    auto u = [&]() {
        z = mix(z);
        return float(z >> 40) * 0x1p-24f;
    };
    const int kind = int(mix(i) % 16);
    const float scale = exp2f(-9.f + 26.f * u());
    e[0] = scale * (0.5f + u());
    e[1] = kind < 6 ? e[0] * (1.f + (u() - 0.5f) * exp2f(-20.f * u())) : exp2f(-9.f + 26.f * u());
    const float fr = exp2f(-24.f + 26.f * u());
    for (int k = 0; k < 2; k++) e[2 + k] = (u() - 0.5f) * fr * e[k] * sqrtf(9.81f * e[k]);
    if (kind < 6) e[3] = e[2] * (1.f + 0.1f * (u() - 0.5f));
    e[4] = -e[0] * (0.5f + u());
    e[5] = kind % 2 ? e[4] + (e[0] - e[1]) * (u() < 0.5f ? 1.f : u()) : -e[1] * (0.5f + u());
    if (kind == 6) e[2] *= exp2f(-140.f * u());
    if (kind == 7) {
        e[3] *= exp2f(-140.f * u());
        if (u() < 0.5f) {  // still water over a flat or uneven bed
            e[1] = e[0];
            e[2] = e[3] * u();
            e[5] = u() < 0.5f ? e[4] : e[4] * (1.f + exp2f(-22.f));
        }
    }
    if (kind == 8) e[2] = u() < 0.5f ? 0.f : -0.f;
    if (kind == 9) e[3] = u() < 0.5f ? 0.f : -0.f;
    if (kind == 8 || kind == 9) e[5] = e[4];
    if (kind == 10) e[0] = u() < 0.3f ? 0.f : 0.02f * u();
    if (kind == 11) e[1] = u() < 0.3f ? 0.f : 0.02f * u();
    if (kind == 12) e[5] = e[4] * (1.f + exp2f(-23.f));
    if (kind == 13) {  // far out of range
        for (int k = 0; k < 6; k++)
            if (u() < 0.3f) e[k] *= exp2f((u() - 0.5f) * 250.f);
        if (u() < 0.1f) e[int(u() * 6.f)] = u() < 0.5f ? INFINITY : NAN;
    }
    if (kind == 14) e[2] *= 1000.f;                 // supersonic
    if (kind == 15) e[3] = -e[3] * exp2f(4.f * u());
}

template <int S> __device__ bool fhDiffers(const float e[6]) {
    Cell L, R, unused;
    cellQuantities<S>(e[0], e[2], 0.f, e[4], L, unused);
    cellQuantities<S>(e[1], e[3], 0.f, e[5], R, unused);
    float a, b, c, d, s;
    edgeFH<S>(L, R, a, b, c, d, s);
    const EdgeOut o = edgeFHGeneral<S>(e[0], e[1], e[2], e[3], e[4], e[5]);
    const float sp = edgeSpeedFH<S>(L, R), sg = edgeSpeedFHGeneral<S>(e[0], e[1], e[2], e[3]);
    return !same(a, o.hL) || !same(b, o.hR) || !same(c, o.huL) || !same(d, o.huR) || !same(s, o.speed) || !same(sp, sg);
}

__global__ void edges(unsigned long long *c, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        float e[6];
        randomEdge(i, e);
        count(c, FWAVE, fhDiffers<SOLVER_FWAVE>(e));
        count(c, HLLE, fhDiffers<SOLVER_HLLE>(e));
        float a, b, p, q, s;
        if (augRieTame(e[0], e[1], e[2], e[3], e[4], e[5], a, b, p, q, s)) {
            const EdgeOut o = edgeAugRieGeneral(e[0], e[1], e[2], e[3], e[4], e[5]);
            count(c, AUG, !same(a, o.hL) || !same(b, o.hR) || !same(p, o.huL) || !same(q, o.huR) || !same(s, o.speed));
            count(c, TAKEN, true);
        }
    }
}

int main() {
    unsigned long long *d, h[NCHECK];
    const uint64_t nq = 1ull << 30, ne = 1ull << 29;
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
    unary<<<152 * 8, 256>>>(d);
    quotients<<<152 * 8, 256>>>(d, nq);
    edges<<<152 * 8, 256>>>(d, ne);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    const char *name[NCHECK] = {"rcp", "sqrt", "div", "div_near", "fwave", "hlle", "augrie", "taken"};
    const unsigned long long samples[NCHECK] = {2ull << 30, 1ull << 30, nq, 3 * nq, ne, ne, h[TAKEN], ne};
    for (int k = 0; k < NCHECK; k++) printf("%s %llu %llu\n", name[k], h[k], samples[k]);
    return 0;
}
