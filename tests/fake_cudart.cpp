// A CUDA runtime without a GPU, for tests of the library's host code: device
// memory is host memory, kernels do nothing, and calls can be told to fail.
#include <cuda_runtime.h>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include "fake_cudart.h"

namespace fake {
std::atomic<long long> device_bytes{0}, device_limit{-1}, host_limit{-1};
std::atomic<int> copies{0}, fail_copy{-1}, stream_syncs{0}, open_copies{0};
static std::mutex lock;
static std::map<void*, size_t> blocks;
static thread_local cudaError_t last = cudaSuccess;

static cudaError_t fails(cudaError_t e)
{
    last = e;
    return e;
}
static cudaError_t take(void** p, size_t bytes)
{
    std::lock_guard<std::mutex> g(lock);
    if (device_limit >= 0 && device_bytes + (long long)bytes > device_limit) return fails(cudaErrorMemoryAllocation);
    *p = calloc(1, bytes ? bytes : 1);
    blocks[*p] = bytes;
    device_bytes += (long long)bytes;
    return cudaSuccess;
}
static cudaError_t give(void* p)
{
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> g(lock);
    auto it = blocks.find(p);
    if (it == blocks.end()) return fails(cudaErrorInvalidValue);
    device_bytes -= (long long)it->second;
    blocks.erase(it);
    free(p);
    return cudaSuccess;
}
}  // namespace fake

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int)
{
    memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    p->sharedMemPerBlockOptin = 232448;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t bytes) { return fake::take(p, bytes); }
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t) { return fake::take(p, bytes); }
cudaError_t cudaFree(void* p) { return fake::give(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return fake::give(p); }
cudaError_t cudaMallocHost(void** p, size_t bytes)
{
    if (fake::host_limit >= 0 && (long long)bytes > fake::host_limit) return fake::fails(cudaErrorMemoryAllocation);
    *p = malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s)
{
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    fake::stream_syncs++;
    fake::open_copies = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError()
{
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*)
{
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (fake::copies++ == fake::fail_copy) return fake::fails(cudaErrorUnknown);
    memcpy(d, s, n);
    fake::open_copies++;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
}
