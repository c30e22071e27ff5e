// Preloaded in front of the CUDA runtime: passes every launch with attributes
// on and counts those of four teams (1024 threads) and of one (256).
#include <dlfcn.h>

#include <cuda_runtime_api.h>

static int counts[2];

extern "C" {
void launchCounts(int *c) {
    for (int i = 0; i < 2; i++) {
        c[i] = counts[i];
        counts[i] = 0;
    }
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
    // (the runtime comes in with the library under test, behind no RTLD_NEXT)
    static const auto next = reinterpret_cast<decltype(&cudaLaunchKernelExC)>(
        dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), "cudaLaunchKernelExC"));
    if (!next) return cudaErrorUnknown;
    counts[0] += c->blockDim.x == 1024;
    counts[1] += c->blockDim.x == 256;
    return next(c, f, args);
}
}
