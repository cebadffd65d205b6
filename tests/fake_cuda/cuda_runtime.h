// The few CUDA runtime calls that csrc/hostcopy.h makes, on the host: copies are
// done at once, and the test sets which calls fail.
#pragma once
#include <cstdlib>
#include <cstring>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
enum { cudaHostAllocDefault = 0, cudaEventDisableTiming = 2 };
struct cudaPointerAttributes { cudaMemoryType type; };
typedef void *cudaStream_t;
typedef void *cudaEvent_t;

namespace fake {
inline thread_local cudaError_t pending = cudaSuccess;
inline cudaMemoryType type = cudaMemoryTypeUnregistered;
inline bool no_attributes = false, no_host_alloc = false;
inline int copies = 0;
inline cudaError_t set(cudaError_t e)
{
    if(e != cudaSuccess) pending = e;
    return e;
}
} // namespace fake

inline cudaError_t cudaGetLastError()
{
    const cudaError_t e = fake::pending;
    fake::pending = cudaSuccess;
    return e;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
    a->type = fake::type;
    return fake::set(fake::no_attributes ? cudaErrorInvalidValue : cudaSuccess);
}
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    ++fake::copies;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    if(fake::no_host_alloc) return fake::set(cudaErrorMemoryAllocation);
    *p = std::malloc(n);
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void *p)
{
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    *e = (void *)1;
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
