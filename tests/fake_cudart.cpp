// A stand-in for the CUDA runtime's calls that the stepping entry points make,
// preloaded in front of the real library: memory is the host's, kernels do not
// run, and every launch leaves a letter in a log -- c: cooperative, r: a
// cooperative one that was refused, k: any other.  Two switches: cooperative
// launches are refused, and every stream belongs to a green context.
#include <cstdlib>
#include <cstring>
#include <string>

#include <cuda.h>
#include <cuda_runtime_api.h>

static std::string launches;
static bool refuse, green;

static CUresult streamGetGreenCtx(CUstream, CUgreenCtx *g) {
    *g = green ? reinterpret_cast<CUgreenCtx>(&green) : nullptr;
    return CUDA_SUCCESS;
}

extern "C" {
void fakeSet(int refuseCooperative, int greenStreams) {
    refuse = refuseCooperative;
    green = greenStreams;
    launches.clear();
}
const char *fakeLaunches() { return launches.c_str(); }

cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *q) {
    const bool known = !strcmp(name, "cuStreamGetGreenCtx");
    *f = known ? reinterpret_cast<void *>(streamGetGreenCtx) : nullptr;
    *q = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    static char scratch[1 << 20];
    *p = scratch;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "an error of the stand-in"; }

cudaError_t __cudaGetKernel(void **k, const void *) { *k = nullptr; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(void *, dim3, dim3, void **, size_t, cudaStream_t) {
    launches += 'k';
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) {
    bool cooperative = false;
    for (unsigned i = 0; i < c->numAttrs; i++)
        cooperative |= c->attrs[i].id == cudaLaunchAttributeCooperative && c->attrs[i].val.cooperative;
    launches += !cooperative ? 'k' : refuse ? 'r' : 'c';
    return cooperative && refuse ? cudaErrorCooperativeLaunchTooLarge : cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t n) { *p = calloc(n + 1, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = reinterpret_cast<cudaStream_t>(0x100); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { launches += '['; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { launches += ']'; *g = nullptr; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(0x200);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { launches += 'g'; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(0x300); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
}
