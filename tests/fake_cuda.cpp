// Stand-ins for the CUDA runtime calls of fm_staging.cu that work on host memory, fail where a
// scenario says so, and count (see staging_paths.cu).
#include "fake_cuda.h"

#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <cstdlib>
#include <cstring>

std::vector<Range> g_ranges;
bool g_no_pinned = false;
int g_threads_left = 1 << 30;
int g_direct = 0, g_staged = 0;

namespace {

std::vector<Range> g_ring;   // what cudaHostAlloc returned

const Range* find(const std::vector<Range>& v, const void* p)
{
    for (const Range& r : v)
        if (static_cast<const char*>(p) >= r.p && static_cast<const char*>(p) < r.p + r.n) return &r;
    return nullptr;
}

}  // namespace

extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    if (g_no_pinned) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    g_ring.push_back(Range{static_cast<char*>(*p), n, cudaMemoryTypeHost});
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
    std::free(p);
    g_ring.clear();
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    const Range* r = find(g_ranges, p);
    a->type = r ? r->type : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t)
{
    const void* host = kind == cudaMemcpyHostToDevice ? src : dst;
    const Range* r = find(g_ranges, host);
    if (r && r->type == cudaMemoryTypeDevice) return cudaErrorInvalidValue;
    ++(find(g_ring, host) ? g_staged : g_direct);
    std::memcpy(dst, src, n);
    return cudaSuccess;
}
int pthread_create(pthread_t* t, const pthread_attr_t* attr, void* (*fn)(void*), void* arg) noexcept
{
    if (g_threads_left <= 0) return EAGAIN;
    --g_threads_left;
    using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    static const Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
    return real(t, attr, fn, arg);
}
// registration of a translation unit's (empty) device code
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaInitModule(void**) {}
}
