// C-ABI: contexts, scene release and ray queries (scene creation: fm_scene_build.cu).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <unordered_map>

#include "fm_internal.h"
#include "fm_staging.h"
#include "fm_trace.cuh"

using namespace fm;

namespace {

constexpr int kQueryBlock = 128, kQueryBlocksPerSm = 8;   // 64 registers per thread

// Large queries: persistent warps over the stream of rays (see trace_stream).  2 M incoherent
// rays through 1.3 M triangles: 958 -> 412 us against one thread per ray; 1 M occlusion rays
// through 20 k triangles: 292 -> 154 us.
__global__ void __launch_bounds__(kQueryBlock, kQueryBlocksPerSm)
k_trace(const QueryRays q, uint32_t n, uint32_t tail, unsigned* next, uint32_t* status)
{
    extern __shared__ float4 s_trace[];
    trace_stream(q, n, next, tail, s_trace, status);
}

// Queries whose rays are all in flight at once: the launch takes as long as its slowest warp,
// so every lane keeps its one ray, and a warp holds only per_warp of them when there are
// fewer rays than lanes (rays of one warp wait for one another's steps).
__global__ void __launch_bounds__(kQueryBlock, kQueryBlocksPerSm)
k_trace_short(const QueryRays q, uint32_t n, uint32_t per_warp, uint32_t* status)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i = (blockIdx.x * (kQueryBlock / 32) + (threadIdx.x >> 5)) * per_warp + lane;
    if (lane >= per_warp || i >= n) return;
    const StreamRay r = q.load(i);
    Hit h;
    if (r.any)
        trace_ray<true>(*r.scene, r.o, r.d, r.tmin, r.tmax, h, status);
    else
        trace_ray<false>(*r.scene, r.o, r.d, r.tmin, r.tmax, h, status);
    q.finish(i, h);
}

}  // namespace

// One ray per lane up to as many rays as lanes can be resident, the stream above.  At that line
// (151,552 rays on 148 SMs) the first form is ahead, as each warp's start and first claim
// cost the stream 5 to 30 us; it falls behind between 200,000 and 300,000 incoherent rays,
// where whole warps wait for their slowest ray a second time, and not at all up to 1 M
// coherent ones.  One ray per lane / stream, us, around a device-pointer call: 20 k
// triangles, random rays, 100 k 76 / 87, 152 k 85 / 96, 200 k 96 / 97, 300 k 120 / 109, 1 M
// 284 / 170; 1.3 M triangles, random, 100 k 158 / 182, 152 k 158 / 172, 300 k 185 / 170, 1 M
// 415 / 256, camera rays 152 k 156 / 180, 300 k 147 / 155, 1 M 183 / 204.
cudaError_t fm::launch_query(cudaStream_t stream, int num_sms, const QueryRays& q, int64_t n, unsigned* next, uint32_t* status)
{
    const int64_t warps = (int64_t)num_sms * kQueryBlocksPerSm * (kQueryBlock / 32);
    if (n <= 32 * warps) {
        const uint32_t per_warp = (uint32_t)((n + warps - 1) / warps);
        const int64_t used = (n + per_warp - 1) / per_warp;
        k_trace_short<<<(int)((used + kQueryBlock / 32 - 1) / (kQueryBlock / 32)), kQueryBlock, 0, stream>>>(q, (uint32_t)n, per_warp, status);
        return cudaGetLastError();
    }
    constexpr int64_t kLaunchRays = (int64_t)1 << 30;   // ray indices are 32-bit within a launch
    for (int64_t first = 0; first < n; first += kLaunchRays) {
        if (first > 0) {
            const cudaError_t e = cudaMemsetAsync(next, 0, sizeof(unsigned), stream);
            if (e != cudaSuccess) return e;
        }
        QueryRays part = q;
        part.rays += 2 * first;
        if (part.occ) part.occ += first;
        if (part.obj) part.obj += first;
        if (part.t) part.t += first;
        k_trace<<<num_sms * kQueryBlocksPerSm, kQueryBlock, kTraceSmemPerThread * kQueryBlock, stream>>>(
            part, (uint32_t)std::min(n - first, kLaunchRays), (uint32_t)(32 * warps), next, status);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

namespace {

fm_status trace_common(fm_ctx* ctx, const fm_scene* sc, const float* rays, int64_t n, int32_t* obj, float* t,
                       uint8_t* occ, int32_t flags)
{
    if (!ctx) return FM_ERR_INVALID;
    if (!sc || n < 0 || (n > 0 && !rays)) return set_error(ctx, FM_ERR_INVALID, "trace: bad arguments");
    if (n == 0) return FM_OK;
    if (!occ && (!obj || !t)) return set_error(ctx, FM_ERR_INVALID, "trace: null output");
    FM_CUDA_TRY(ctx, cudaSetDevice(ctx->device), "cudaSetDevice");
    const bool dev = (flags & FM_FLAG_DEVICE_PTRS) != 0;
    const float* d_rays = rays;
    int32_t* d_obj = obj;
    float* d_t = t;
    uint8_t* d_occ = occ;
    void* tmp = nullptr;
    if (!dev) {
        const size_t bytes = 32 * (size_t)n + (occ ? (size_t)n : 8 * (size_t)n);
        FM_CUDA_TRY(ctx, cudaMallocAsync(&tmp, bytes, ctx->stream), "trace alloc");
        char* p = static_cast<char*>(tmp);
        d_rays = reinterpret_cast<float*>(p);
        FM_CUDA_TRY(ctx, copy_in(ctx, ctx->stream, {InCopy{p, rays, 32 * (size_t)n}}), "trace h2d");
        p += 32 * (size_t)n;
        if (occ) {
            d_occ = reinterpret_cast<uint8_t*>(p);
        } else {
            d_obj = reinterpret_cast<int32_t*>(p);
            d_t = reinterpret_cast<float*>(p + 4 * (size_t)n);
        }
    }
    // the status word and, in the same allocation, the query's ray counter
    FM_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_status, 0, 64, ctx->stream), "trace");
    const QueryRays q{reinterpret_cast<const float4*>(d_rays), sc->d_dev, d_obj, d_t, d_occ};
    FM_CUDA_TRY(ctx, launch_query(ctx->stream, ctx->num_sms, q, n, ctx->d_status + 8, ctx->d_status), "trace launch");
    if (!dev) {
        if (occ)
            FM_CUDA_TRY(ctx, copy_results(ctx, ctx->stream, {OutCopy{occ, d_occ, (size_t)n}}), "trace d2h");
        else
            FM_CUDA_TRY(ctx, copy_results(ctx, ctx->stream, {OutCopy{obj, d_obj, 4 * (size_t)n}, OutCopy{t, d_t, 4 * (size_t)n}}), "trace d2h");
        FM_CUDA_TRY(ctx, cudaFreeAsync(tmp, ctx->stream), "trace free");
    }
    uint32_t status = 0;
    FM_CUDA_TRY(ctx, cudaMemcpyAsync(&status, ctx->d_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream),
                "status");
    FM_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "trace sync");
    if (status & 1u) return set_error(ctx, FM_ERR_QUEUE_OVERFLOW, "trace: traversal stack overflow");
    return FM_OK;
}

}  // namespace

extern "C" {

fm_status fm_ctx_create(int device, fm_ctx** out)
{
    if (!out) return FM_ERR_INVALID;
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) return FM_ERR_NO_DEVICE;
    if (device < 0 || device >= count) return FM_ERR_INVALID;
    fm_ctx* ctx = new (std::nothrow) fm_ctx();
    if (!ctx) return FM_ERR_OOM;
    ctx->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&ctx->d_status, 64) != cudaSuccess) {
        delete ctx;
        return FM_ERR_CUDA;
    }
    cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device);
    // Scenes, BVH builds and renders allocate from the device's default memory pool with
    // stream-ordered calls; keeping freed blocks in the pool makes creating and
    // destroying scenes cheap (no release to the driver at every synchronisation).
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
        uint64_t keep = UINT64_MAX;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    *out = ctx;
    return FM_OK;
}

void fm_ctx_destroy(fm_ctx* ctx)
{
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    fm::scene_builder_release(ctx);
    fm::staging_release(ctx);
    fm::wf_cache_release(ctx);
    cudaFree(ctx->d_status);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}

const char* fm_last_error(const fm_ctx* ctx) { return ctx ? ctx->error.c_str() : "null context"; }

// Used by the host-side scene loader (compiled by the C++ compiler) to report errors.
void fm_internal_set_error(fm_ctx* ctx, const char* msg)
{
    if (ctx) ctx->error = msg ? msg : "";
}

fm_status fm_scene_destroy(fm_ctx* ctx, fm_scene* sc)
{
    if (!ctx) return FM_ERR_INVALID;
    if (!sc) return FM_OK;
    cudaSetDevice(ctx->device);
    for (void* p : sc->allocations) cudaFreeAsync(p, ctx->stream);
    sc->shared_bvh.reset();   // frees the BVH arrays when no other scene of its group holds them
    cudaStreamSynchronize(ctx->stream);
    delete sc;
    return FM_OK;
}

fm_status fm_scene_bvh_stats(fm_ctx* ctx, const fm_scene* sc, int64_t* nodes, int64_t* prims, int32_t* depth,
                             double* build_ms)
{
    if (!ctx) return FM_ERR_INVALID;
    if (!sc) return set_error(ctx, FM_ERR_INVALID, "bvh_stats: null scene");
    if (nodes) *nodes = sc->bvh.num_nodes;
    if (prims) *prims = sc->bvh.num_leaf;
    if (depth) *depth = sc->bvh.depth;
    if (build_ms) *build_ms = sc->bvh.build_ms;
    return FM_OK;
}

fm_status fm_trace_closest(fm_ctx* ctx, const fm_scene* scene, const float* rays, int64_t n, int32_t* obj_id, float* t,
                           int32_t flags)
{
    return trace_common(ctx, scene, rays, n, obj_id, t, nullptr, flags);
}

fm_status fm_trace_any(fm_ctx* ctx, const fm_scene* scene, const float* rays, int64_t n, uint8_t* occluded,
                       int32_t flags)
{
    if (!occluded && n > 0) return ctx ? set_error(ctx, FM_ERR_INVALID, "trace_any: null output") : FM_ERR_INVALID;
    return trace_common(ctx, scene, rays, n, nullptr, nullptr, occluded, flags);
}

}  // extern "C"
