// A CUDA runtime without a GPU for host-logic tests: two devices with their own
// attributes, "device" memory on the host, streams that are always idle.
// Defined in the test's executable, these take the place of libcudart's
// functions in libtsuner_b200.so.  Kernels do not run; their launches are
// checked against the attributes that the current device was given and kept.
#pragma once
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace fake {
struct Launch {
    int device;
    unsigned grid;
    size_t smem;
};
inline std::mutex mu;
inline thread_local int device = 0;
inline thread_local cudaError_t last = cudaSuccess;  // of a launch or an allocation
inline int sms[2] = {148, 100};
inline std::map<std::pair<int, const void *>, int> smem_limit;  // (device, kernel) -> attribute
inline std::vector<Launch> launches;
inline std::map<void *, size_t> blocks;  // live allocations
inline size_t in_use = 0, memory = ~(size_t)0, peak = 0;
inline thread_local dim3 cfg_grid, cfg_block;
inline thread_local size_t cfg_smem;
inline thread_local cudaStream_t cfg_stream;

inline cudaError_t alloc(void **p, size_t n) {
    std::lock_guard<std::mutex> g(mu);
    if (in_use + n > memory) return last = cudaErrorMemoryAllocation;
    *p = std::calloc(1, n ? n : 1);
    blocks[*p] = n;
    in_use += n;
    if (in_use > peak) peak = in_use;
    return cudaSuccess;
}
inline cudaError_t release(void *p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> g(mu);
    auto it = blocks.find(p);
    if (it == blocks.end()) return cudaErrorInvalidValue;
    in_use -= it->second;
    blocks.erase(it);
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t launch(const void *k, dim3 grid, size_t smem) {
    std::lock_guard<std::mutex> g(mu);
    auto it = smem_limit.find({device, k});
    if (smem > 48 * 1024 && (it == smem_limit.end() || (size_t)it->second < smem))
        return last = cudaErrorInvalidValue;
    launches.push_back({device, grid.x * grid.y * grid.z, smem});
    return cudaSuccess;
}
inline CUresult encode(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                       const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return CUDA_SUCCESS;
}
inline cudaError_t rows(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h) {
    for (size_t r = 0; r < h; r++) std::memcpy((char *)d + r * dp, (const char *)s + r * sp, w);
    return cudaSuccess;
}
}  // namespace fake

extern "C" {
void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st *st) {
    fake::cfg_grid = g;
    fake::cfg_block = b;
    fake::cfg_smem = s;
    fake::cfg_stream = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
    *g = fake::cfg_grid;
    *b = fake::cfg_block;
    *s = fake::cfg_smem;
    *(cudaStream_t *)st = fake::cfg_stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *k, dim3 g, dim3, void **, size_t s, cudaStream_t) { return fake::launch(k, g, s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *k, void **) {
    return fake::launch(k, c->gridDim, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void *k, cudaFuncAttribute a, int v) {
    std::lock_guard<std::mutex> g(fake::mu);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) fake::smem_limit[{fake::device, k}] = v;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d > 1) return cudaErrorInvalidDevice;
    fake::device = d;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = fake::device;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int d) {
    *v = a == cudaDevAttrMultiProcessorCount ? fake::sms[d] : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMalloc(void **p, size_t n) { return fake::alloc(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return fake::alloc(p, n); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return fake::alloc(p, n); }
cudaError_t cudaFree(void *p) { return fake::release(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return fake::release(p); }
cudaError_t cudaMallocHost(void **p, size_t n) {
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void *p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) {
    *p = (cudaMemPool_t)1;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    return fake::rows(d, dp, s, sp, w, h);
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void *d, const void *, size_t n, size_t, cudaMemcpyKind) {
    std::memset(d, 0, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    std::memset(a, 0, sizeof(*a));
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *, void **f, unsigned long long, cudaDriverEntryPointQueryResult *q) {
    *f = (void *)fake::encode;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = (cudaEvent_t)1;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.f;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = (cudaStream_t)8;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) {
    *c = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
}
