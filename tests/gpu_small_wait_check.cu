// The small domain's step kernel where a meeting's wait runs out: the meeting
// point is set up for one CTA more than is launched.  Prints a line per run:
// name, status bits, dt, NaN depths written, depths left alone, whether the
// input changed, milliseconds.
#include <cmath>
#include <cstdio>
#include <vector>

#include "swe_small.cu"

using namespace swegb;

constexpr int NX = 3, NY = 40, P = NY + 2, N = (NX + 2) * P, ROWS = 64;

int main() {
    float *q[8];  // h, hu, hv twice, b
    for (float *&p : q)
        if (cudaMalloc(&p, N * 4) != cudaSuccess || cudaMemset(p, 0, N * 4) != cudaSuccess) return 2;
    std::vector<float> h(N), out(N), in(N);
    for (int i = 0; i < N; i++) h[i] = 2.f + 0.01f * (i % 7);
    BlockDesc B{};
    B.nx = NX; B.ny = NY; B.pitch = P; B.dx = B.dy = 1.f;
    for (int k = 0; k < 4; k++) { B.bnd[k] = WALL; B.nbr[k] = -1; }
    std::vector<WorkUnit> u;
    for (int x = 1; x <= NX; x++) u.push_back(WorkUnit{0, 1, x, x + 1});
    BlockDesc *dB; WorkUnit *dU; GroupState *dG; small::Sync *dY;
    if (cudaMalloc(&dB, sizeof(B)) || cudaMalloc(&dU, sizeof(WorkUnit) * NX) || cudaMalloc(&dG, sizeof(GroupState)) ||
        cudaMalloc(&dY, sizeof(small::Sync)))
        return 2;
    cudaMemcpy(dB, &B, sizeof(B), cudaMemcpyHostToDevice);
    cudaMemcpy(dU, u.data(), sizeof(WorkUnit) * NX, cudaMemcpyHostToDevice);
    DomainDev d{};
    d.h[0] = q[0]; d.hu[0] = q[1]; d.hv[0] = q[2]; d.h[1] = q[3]; d.hu[1] = q[4]; d.hv[1] = q[5]; d.b = q[6];
    d.blocks = dB; d.units = dU; d.groups = dG; d.nblocks = 1;
    d.solver = SOLVER_HLLE; d.semantics = SEM_UNSPLIT;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const char *name[3] = {"meets", "runs_out", "again"};
    for (int run = 0; run < 3; run++) {
        if (run < 2) {
            GroupState G{};
            G.enabled = 1;
            G.target = INFINITY;
            const small::Sync Y{0u, 0u, 0ull, run ? NX + 1 : NX, 0};
            cudaMemcpy(dG, &G, sizeof(G), cudaMemcpyHostToDevice);
            cudaMemcpy(dY, &Y, sizeof(Y), cudaMemcpyHostToDevice);
        }
        for (int i = 0; i < N; i++) out[i] = -1.f;
        cudaMemcpy(q[0], h.data(), N * 4, cudaMemcpyHostToDevice);
        cudaMemcpy(q[3], out.data(), N * 4, cudaMemcpyHostToDevice);
        cudaEventRecord(e0);
        if (small::launch(d, dU, NX, dY, 1, 1, ROWS, nullptr) != cudaSuccess) return 3;
        cudaEventRecord(e1);
        if (cudaDeviceSynchronize() != cudaSuccess) return 4;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        GroupState G;
        cudaMemcpy(&G, dG, sizeof(G), cudaMemcpyDeviceToHost);
        cudaMemcpy(out.data(), q[3], N * 4, cudaMemcpyDeviceToHost);
        cudaMemcpy(in.data(), q[0], N * 4, cudaMemcpyDeviceToHost);
        int nans = 0, left = 0, changed = 0;
        for (int x = 1; x <= NX; x++)
            for (int y = 1; y <= NY; y++) {
                nans += std::isnan(out[x * P + y]);
                left += out[x * P + y] == -1.f;
            }
        for (int i = 0; i < N; i++) changed += in[i] != h[i];
        printf("%s %d %g %d %d %d %g\n", name[run], G.status, double(G.dt), nans, left, changed, double(ms));
    }
    return 0;
}
