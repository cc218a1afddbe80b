// Warps that traverse a stream of rays: the loop of the wavefront's trace kernel and of large ray
// queries.
//
// The loop is bound by instruction issue, so it is arranged to run every part of a
// traversal with as many of the warp's lanes as possible:
//  * Rays are set up (loads, reciprocals, shear: about 250 instructions) by the whole warp,
//    32 at a time, into shared memory; a lane whose query completes picks the next
//    prepared ray up with four 16-byte reads.  A lane in six completes per step, so
//    setting a ray up in the lane that needs it ran that code for six lanes at a time.
//  * A pass of the loop visits one node in the lanes without pending primitives, then tests
//    primitives one at a time while enough lanes have any (kPrimWait).  Finishing every
//    lane's primitives before the next node ran the test 2.6 times per node at 6.9 lanes; now
//    it runs 1.4 times at 12.6.
// A lane never visits a node before its own pending primitives are tested, so each ray sees
// the nodes and primitives in the order, and with the t_best, of a plain traversal: hits do
// not depend on what the other lanes do, near ties included.
// Measured with the 16-scene batch (241 M rays; 2^24 path slots): 42.8 -> 27.7 ms of trace
// time per render; the 1.3 M-triangle mesh at 1920x1080: 4.61 -> 3.29 ms.  Per 32 rays the warp
// runs 5.7 node steps, 8.2 primitive steps, 5.3 pick-ups and 1.03 set-ups.
#pragma once
#include "fm_bvh.cuh"

namespace fm {

// Stack entries per thread kept in shared memory (the rest in local memory): 2 / 4 / 6
// entries traced the 16-scene batch in 29.4 / 29.1 / 29.1 ms.
constexpr int kTraceSmemStack = 4;
// Pending primitives are tested again and again until at most kPrimWait lanes have any and
// more than kNodeReady lanes can visit their next node: the last few lanes' tests then run
// together with those of that node.  Never waiting (0) traced the batch in 32.4 ms,
// 4 / 8 / 12 / 16 / 31 lanes in 29.5 / 29.3 / 29.8 / 30.3 / 30.6 ms.  kNodeReady 6 to 15 made no
// difference there; counting lanes that wait for a new ray as ready slowed a scene of a
// single node (Cornell box: 0.44 against 0.40 ms), whose lanes it pulled out of step.
constexpr int kPrimWait = 8;
constexpr int kNodeReady = 6;
// Dynamic shared memory per thread of trace_stream: stack entries and one prepared ray.
constexpr size_t kTraceSmemPerThread = sizeof(uint2) * kTraceSmemStack + 4 * sizeof(float4);

// A ray as its source hands it over.
struct StreamRay {
    f3 o, d;
    float tmin, tmax;
    bool any;              // occlusion query
    const DevScene* scene;
};

// Traces rays [0, total) of `src`, shared by all warps of the grid through *next (0 before
// the launch).  `src` provides
//   StreamRay load(uint32_t idx)                       the ray (called by up to 32 lanes at once)
//   float tmin(uint32_t idx, bool any)                  its t_min alone
//   void finish(uint32_t idx, const Hit& h)            its result
// (a lane that meets a sphere's box loads its ray again).
// Within `tail` rays of the end a warp claims only what its idle lanes need, so that no warp
// holds back rays while others run dry.  Call with all threads of the block; smem holds
// kTraceSmemPerThread bytes per thread.
template <class Src>
FM_D void trace_stream(const Src& src, uint32_t total, unsigned* next, uint32_t tail, void* smem, uint32_t* status)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int nthr = blockDim.x;
    SharedTopStack<kTraceSmemStack> stack;
    // prepared rays: four 16-byte columns, one entry per thread, each warp its own 32
    float4* const col = static_cast<float4*>(smem) + (threadIdx.x - lane);
    stack.top = reinterpret_cast<uint2*>(static_cast<float4*>(smem) + 4 * nthr) + threadIdx.x;
    stack.stride = nthr;
    uint32_t head = 0, avail = 0;       // the warp's prepared rays not yet picked up
    bool more = true;                   // rays may be left to claim
    bool whole = tail < total;          // claim whole warps of rays
    // this lane's ray
    bool live = false, any = false;
    RayTrav r{};
    float tmin = 0.0f;
    Hit hit{0.0f, -1, 0.0f, 0.0f};      // hit.t: t_best
    uint32_t idx = 0;
    int sp = 0;
    uint2 group = make_uint2(0u, 0u);
    uint32_t pbase = 0, pmask = 0, lmask = 0;   // primitives of the last visited node still to test
    const uint4* nodes = nullptr;
    const float4* leaf = nullptr;
    for (;;) {
        const bool fin = live && pmask == 0u && group.y <= 0x00ffffffu && sp == 0;
        const unsigned idle = __ballot_sync(0xffffffffu, !live || fin);
        if (idle) {
            if (fin) {
                src.finish(idx, hit);
                live = false;
            }
            if (avail == 0 && more) {
                const uint32_t take = whole ? 32u : (uint32_t)__popc(idle);
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(next, take);
                base = __shfl_sync(0xffffffffu, base, 0);
                whole = whole && total - min(base, total) > tail;
                const uint32_t end = min(base + take, total);
                avail = base < end ? end - base : 0u;
                more = base + take < total;
                head = 0;
                // the warp's rays of the previous claim have all been picked up
                __syncwarp();
                if ((uint32_t)lane < avail) {
                    const StreamRay q = src.load(base + lane);
                    const RayTrav t = ray_trav(q.o, q.d);
                    const uint32_t f = t.flags | (q.any ? 32u : 0u) | (q.scene->num_nodes == 0 ? 64u : 0u);
                    col[lane] = make_float4(t.no.x, t.no.y, t.no.z, q.tmax);
                    col[nthr + lane] = make_float4(t.idir.x, t.idir.y, t.idir.z, __uint_as_float(f));
                    col[2 * nthr + lane] = make_float4(t.sx, t.sy, t.sz, __uint_as_float(base + lane));
                    const unsigned long long pn = (unsigned long long)q.scene->nodes, pl = (unsigned long long)q.scene->leaf;
                    reinterpret_cast<ulonglong2*>(col)[3 * nthr + lane] = make_ulonglong2(pn, pl);
                }
                __syncwarp();
            }
            const uint32_t rank = (uint32_t)__popc(idle & lt);
            if (!live && rank < avail) {
                const uint32_t e = head + rank;
                const float4 a = col[e], b = col[nthr + e], c = col[2 * nthr + e];
                const ulonglong2 p = reinterpret_cast<const ulonglong2*>(col)[3 * nthr + e];
                const uint32_t f = __float_as_uint(b.w);
                r = RayTrav{f3{a.x, a.y, a.z}, f3{b.x, b.y, b.z}, c.x, c.y, c.z, f & 31u};
                idx = __float_as_uint(c.w);
                any = (f & 32u) != 0u;
                hit = Hit{a.w, -1, 0.0f, 0.0f};
                tmin = src.tmin(idx, any);
                nodes = reinterpret_cast<const uint4*>(p.x);
                leaf = reinterpret_cast<const float4*>(p.y);
                group = root_group(1, f & 7u);
                sp = 0;
                pmask = 0u;
                live = (f & 64u) == 0u;
                if (!live) src.finish(idx, hit);   // an empty scene
            }
            const uint32_t taken = min((uint32_t)__popc(idle), avail);
            head += taken;
            avail -= taken;
            if (__ballot_sync(0xffffffffu, live) == 0u) {
                if (avail == 0 && !more) break;
                continue;
            }
        }
        // node step
        if (live && pmask == 0u) {
            if (group.y <= 0x00ffffffu) group = stack.get(--sp);
            const uint32_t child = next_child(group, ray_octant(r), sp, stack, status);
            const NodeHits h = intersect_node(nodes + 5 * (size_t)child, r, tmin, hit.t);
            group = make_uint2(h.child_base, h.node_bits);
            pbase = h.prim_base;
            pmask = h.prim_bits;
            lmask = h.lmask;
        }
        // primitive steps
        for (;;) {
            const unsigned pending = __ballot_sync(0xffffffffu, live && pmask != 0u);
            if (__popc(pending) <= kPrimWait) {
                if (pending == 0u) break;
                const bool ready = live && pmask == 0u && (group.y > 0x00ffffffu || sp > 0);
                if (__popc(__ballot_sync(0xffffffffu, ready)) > kNodeReady) break;
            }
            if (live && pmask != 0u) {
                const uint32_t below = (pmask & (0u - pmask)) - 1u;
                const float4* rec = leaf + 3 * (size_t)(pbase + __popc(lmask & below));
                pmask &= pmask - 1u;
                auto sphere = [&](int i, float& t) {
                    const StreamRay q = src.load(idx);
                    const SphereDev& s = q.scene->spheres[i];
                    return intersect_sphere(s.w2o, s.radius, q.o, q.d, tmin, hit.t, t);
                };
                if (test_prim(rec, r, tmin, hit.t, hit, any, sphere) && any) {
                    pmask = 0u;
                    group.y = 0u;
                    sp = 0;
                }
            }
        }
    }
}

// The rays of a query as a stream: n x 8 floats (origin, t_min, direction, t_max) against one
// scene; results as fm_trace_closest / fm_trace_any return them.
struct QueryRays {
    const float4* rays;
    const DevScene* scene;
    int32_t* obj;
    float* t;
    uint8_t* occ;   // null: closest hits
    FM_D StreamRay load(uint32_t idx) const
    {
        const float4 a = __ldg(rays + 2 * (size_t)idx), b = __ldg(rays + 2 * (size_t)idx + 1);
        return StreamRay{f3{a.x, a.y, a.z}, f3{b.x, b.y, b.z}, a.w, b.w, occ != nullptr, scene};
    }
    FM_D float tmin(uint32_t idx, bool) const { return __ldg(&rays[2 * (size_t)idx].w); }
    FM_D void finish(uint32_t idx, const Hit& h) const
    {
        if (occ) {
            occ[idx] = h.prim >= 0 ? 1 : 0;
        } else {
            obj[idx] = h.prim >= 0 ? __ldg(scene->prim_obj + h.prim) : -1;
            t[idx] = h.prim >= 0 ? h.t : __int_as_float(0x7f800000);
        }
    }
};

// Traces q's n rays; next and status are device words, zero before the launch.
cudaError_t launch_query(cudaStream_t stream, int num_sms, const QueryRays& q, int64_t n, unsigned* next, uint32_t* status);

}  // namespace fm
