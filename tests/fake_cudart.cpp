// A stand-in for the calls of the CUDA runtime that matrices, problems and
// densities are made and freed with, for tests that need two devices or none:
// preloaded before the library, it counts two devices, hands out host memory
// and launches nothing.  It keeps each allocation's device and whether that
// device was waited for since; fake_report() counts the frees that cudaFreeAsync
// would get wrong.  fake_launches() counts the launches, and fake_refuse() makes
// those with attributes (clusters) fail.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>

namespace {
struct Block {
    int device;
    bool waited;
};
std::map<void*, Block> blocks;
std::map<cudaMemPool_t, int> pools;
int current = 0, wrong_device = 0, not_waited = 0;
int plain = 0, extended = 0, refuse = 0, plain_blocks = 0;
cudaError_t last = cudaSuccess;
}  // namespace

extern "C" {

void fake_report(int* live, int* wrong, int* early, int* cur) {
    *live = (int)blocks.size();
    *wrong = wrong_device;
    *early = not_waited;
    *cur = current;
}

int fake_plain_blocks() { return plain_blocks; }
void fake_refuse(int on) { refuse = on; }
void fake_launches(int* p, int* x) {
    *p = plain;
    *x = extended;
}

cudaError_t cudaGetDeviceCount(int* n) { return *n = 2, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = current, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return current = d, cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    return last = cudaSuccess, e;
}
cudaError_t cudaPeekAtLastError() { return last; }

cudaError_t cudaDeviceSynchronize() {
    for (auto& b : blocks)
        if (b.second.device == current) b.second.waited = true;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)malloc(8), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)malloc(8), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }

// plain allocations of 64 MiB and more are counted with the pools' blocks
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = calloc(1, n);
    if (n >= (size_t)64 << 20) {
        blocks[*p] = Block{current, false};
        plain_blocks++;
    }
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) { return blocks.erase(p), free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return memcpy(d, s, n), cudaSuccess;
}

cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* prop) {
    *p = (cudaMemPool_t)malloc(8);
    pools[*p] = prop->location.id;
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { return pools.erase(p), cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
    *p = calloc(1, n);
    blocks[*p] = Block{pools.at(pool), false};
    return cudaSuccess;
}
// on the default stream, whose device is the current one, the memory of another
// device is refused, and work on other streams has to have been waited for
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
    const Block b = blocks.at(p);
    if (s == nullptr || s == cudaStreamLegacy) {
        if (b.device != current) return wrong_device++, cudaErrorInvalidValue;
        if (!b.waited) not_waited++;
    }
    blocks.erase(p);
    free(p);
    return cudaSuccess;
}

cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    return *n = 1, cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return plain++, 1; }  // no launch
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) {
    if (refuse) return last = cudaErrorInvalidClusterSize;
    return extended++, cudaSuccess;
}

}  // extern "C"
