// A CUDA runtime of host memory: allocations are malloc, copies happen at
// once, and the test may make one fail.  For the engine's host code alone; the
// device functions of its headers are declared, never called.
#pragma once

#include <atomic>
#include <chrono>
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <thread>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __align__(n) alignas(n)

struct uint2 { unsigned x, y; };
struct uint4 { unsigned x, y, z, w; };
inline uint2 make_uint2(unsigned x, unsigned y) { return {x, y}; }

enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2, cudaMemcpyDeviceToDevice = 3 };
enum { cudaMemoryTypeUnregistered = 0, cudaMemAllocationTypePinned = 1, cudaMemLocationTypeDevice = 1,
       cudaMemPoolAttrReleaseThreshold = 4 };
enum { cudaEventDisableTiming = 2, cudaHostAllocDefault = 0, cudaStreamNonBlocking = 1 };
using cudaStream_t = struct FakeStream *;
using cudaEvent_t = struct FakeEvent *;
using cudaMemPool_t = struct FakePool *;
struct cudaPointerAttributes { int type; };
struct cudaMemPoolProps { int allocType; struct { int type, id; } location; };

namespace fake {
inline thread_local cudaError_t last = cudaSuccess;
inline std::function<bool()> copy_fails;  // asked by each asynchronous copy
inline std::function<bool(size_t)> pool_refuses;  // asked by each allocation from the pool
inline std::function<bool(size_t)> malloc_refuses;  // and by each other one
inline std::atomic<long> pool_bytes{0};
inline cudaError_t result(bool ok, cudaError_t e = cudaErrorUnknown) {
    if (!ok) last = e;
    return ok ? cudaSuccess : e;
}
}  // namespace fake

inline cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
namespace fake {
inline thread_local int device = 0;
}
inline cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
inline cudaError_t cudaGetDevice(int *d) { *d = fake::device; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d) { fake::device = d; return cudaSuccess; }

template <class T>
cudaError_t cudaMalloc(T **p, size_t n) {
    *p = fake::malloc_refuses && fake::malloc_refuses(n) ? nullptr : static_cast<T *>(std::calloc(1, n ? n : 1));
    return fake::result(*p != nullptr, cudaErrorMemoryAllocation);
}
inline cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
inline cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
inline cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) {
    if (fake::pool_refuses && fake::pool_refuses(n)) return fake::result(false, cudaErrorMemoryAllocation);
    size_t *h = static_cast<size_t *>(std::calloc(1, n + 64));
    if (!h) return fake::result(false, cudaErrorMemoryAllocation);
    *h = n;
    fake::pool_bytes += (long)n;
    *p = reinterpret_cast<uint8_t *>(h) + 64;
    return cudaSuccess;
}
inline cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
    if (!p) return cudaSuccess;
    size_t *h = reinterpret_cast<size_t *>(static_cast<uint8_t *>(p) - 64);
    fake::pool_bytes -= (long)*h;
    std::free(h);
    return cudaSuccess;
}
inline cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { *p = nullptr; return cudaSuccess; }
inline cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, int, void *) { return cudaSuccess; }
inline cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }

inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t = nullptr) {
    if (fake::copy_fails && fake::copy_fails()) return fake::result(false);
    std::memmove(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k); }
inline cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t = nullptr) {
    std::memset(d, v, n);
    return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}

inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return cudaMalloc(s, 8); }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { return cudaFree(s); }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
inline cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaMalloc(e, 8); }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaMalloc(e, 8); }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { return cudaFree(e); }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t = nullptr) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }

// what the headers' device functions name
struct FakeDim { unsigned x; };
extern FakeDim threadIdx, blockIdx, blockDim, gridDim;
int __popc(unsigned);
int __ffs(int);
int __clzll(long long);
void __nanosleep(unsigned);
void __syncthreads();
size_t __cvta_generic_to_shared(const void *);
unsigned __ballot_sync(unsigned, int);
int __any_sync(unsigned, int);
template <class T> T __shfl_up_sync(unsigned, T, int);
template <class T> T __shfl_xor_sync(unsigned, T, int);
template <class T> T atomicOr(T *, T);
template <class T> T atomicAdd(T *, T);
inline uint32_t atomicOr(uint32_t *, int);
