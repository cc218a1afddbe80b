// 8-wide compressed BVH: node format and traversal.
//
// Node (80 bytes = 5 x uint4), one per internal node of the wide tree:
//   w0: origin p.xyz (float), byte-packed [ex, ey, ez, imask]
//   w1: child_base, prim_base, lmask, unused
//   w2: qlo_x[0..7], qlo_y[0..7]      w3: qlo_z[0..7], qhi_x[0..7]
//   w4: qhi_y[0..7], qhi_z[0..7]
// Child i's box is p + q * 2^(e-127) per axis; the quantized box is rounded outward, so
// it always contains the exact box.  imask bit i marks child i as an internal node; the
// internal children are stored contiguously from child_base in slot order.  A leaf child
// holds 1-3 primitives: bits 3i .. 3i+2 of lmask, set from the lowest up; the node's
// primitives are stored contiguously from prim_base in the order of those bits.  An empty
// slot has neither, so its box (all zero) needs no test of its own.
//
// Slots are assigned by octant of the child's centroid relative to the node centre at
// build time, so that visiting slots in the order key = slot ^ ray_octant (highest
// first) is approximately front to back.
//
// Traversal keeps a short stack of node groups (child_base, hit bits << 24 | imask),
// one entry per tree level at most.  The stack is an accessor type: a plain per-thread
// array (LocalStack), or one whose top entries live in shared memory (SharedTopStack),
// which keeps the traversal's most frequent stack traffic out of the L1 cache that holds
// the nodes.
#pragma once
#include "fm_common.cuh"
#include "fm_scene.cuh"
#include "fm_triangle.cuh"

namespace fm {

constexpr int kTraversalStack = 32;   // the builder rejects trees deeper than this
constexpr uint32_t kSphereFlag = 0x80000000u;

struct Hit {
    float t;
    int32_t prim;   // -1 on a miss
    float b1, b2;   // barycentrics of v1 and v2 (triangles)
};

// What a traversal needs of a ray, computed once per ray.
struct RayTrav {
    f3 no;            // negated origin
    f3 idir;          // 1 / direction (components below 1e-20 replaced by +-1e-20)
    float sx, sy, sz; // shear of the triangle test
    uint32_t flags;   // bits 0-2: octant (sign of each direction component), bits 3-4: main axis
};

FM_D uint32_t ray_octant(const RayTrav& r) { return r.flags & 7u; }
FM_D int ray_axis(const RayTrav& r) { return (int)((r.flags >> 3) & 3u); }

FM_D RayTrav ray_trav(f3 o, f3 d)
{
    RayTrav r;
    r.no = -o;
    const float sdx = fabsf(d.x) < 1e-20f ? copysignf(1e-20f, d.x) : d.x;
    const float sdy = fabsf(d.y) < 1e-20f ? copysignf(1e-20f, d.y) : d.y;
    const float sdz = fabsf(d.z) < 1e-20f ? copysignf(1e-20f, d.z) : d.z;
    r.idir = f3{1.0f / sdx, 1.0f / sdy, 1.0f / sdz};
    const RayPre p = ray_pre(d);
    r.sx = p.sx;
    r.sy = p.sy;
    r.sz = p.sz;
    r.flags = (d.x >= 0.0f ? 1u : 0u) | (d.y >= 0.0f ? 2u : 0u) | (d.z >= 0.0f ? 4u : 0u) | (uint32_t)p.kz << 3;
    return r;
}

FM_D float byte_f(uint32_t w, int k) { return (float)((w >> (8 * k)) & 0xffu); }

// Bytes k and k + 1 of w as floats, by conversion instructions (byte_pair) or by placing
// them in the mantissa of 2^23 and subtracting it (byte_pair_alu; exact).  The conversions
// run on a pipe an eighth as wide as a warp: all 48 of a node test there kept it 65 % busy,
// and the other form costs half an instruction more per byte.  Converting one axis and
// placing two traced the 16-scene batch in 28.2 ms against 29.4 (48 conversions) and 28.6
// (none), the 1.3 M-triangle mesh in 3.26 ms against 3.52 and 3.36.
FM_D f32x2 byte_pair(uint32_t w, int k) { return pack2(byte_f(w, k), byte_f(w, k + 1)); }
FM_D f32x2 byte_pair_alu(uint32_t w, int k)
{
    const float a = __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7440u + (unsigned)k));
    const float b = __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7441u + (unsigned)k));
    return add2(pack2(a, b), pack2(-8388608.0f, -8388608.0f));
}

// What a visited node adds to a traversal: the internal children hit (hit bits << 24,
// keyed by slot ^ octant, | imask) and the leaf primitives hit (lmask's layout).
struct NodeHits {
    uint32_t child_base, node_bits, prim_base, prim_bits, lmask;
};

// Intersects the 8 children of a node.  Two children are tested at a time: their plane
// distances per axis and side are one packed multiply-add.
FM_D NodeHits intersect_node(const uint4* __restrict__ np, const RayTrav& r, float tmin, float tmax)
{
    const uint4 w0 = __ldg(np + 0);
    const uint4 w1 = __ldg(np + 1);
    const uint4 w2 = __ldg(np + 2);
    const uint4 w3 = __ldg(np + 3);
    const uint4 w4 = __ldg(np + 4);
    const uint32_t ex = w0.w & 0xffu, ey = (w0.w >> 8) & 0xffu, ez = (w0.w >> 16) & 0xffu;
    const uint32_t imask = w0.w >> 24;
    const float ax = __uint_as_float(ex << 23) * r.idir.x;
    const float ay = __uint_as_float(ey << 23) * r.idir.y;
    const float az = __uint_as_float(ez << 23) * r.idir.z;
    const float bx = (__uint_as_float(w0.x) + r.no.x) * r.idir.x;
    const float by = (__uint_as_float(w0.y) + r.no.y) * r.idir.y;
    const float bz = (__uint_as_float(w0.z) + r.no.z) * r.idir.z;
    const f32x2 ax2 = pack2(ax, ax), ay2 = pack2(ay, ay), az2 = pack2(az, az);
    const f32x2 bx2 = pack2(bx, bx), by2 = pack2(by, by), bz2 = pack2(bz, bz);
    // Near and far planes per axis chosen once per node from the ray's direction signs
    // (t = q a + b grows with q when a = 2^e / d >= 0), so the per-child slab test needs
    // no min / max to order the two planes.  Equal to min / max of the two plane
    // distances, so the results do not change.
    const bool px = r.idir.x >= 0.0f, py = r.idir.y >= 0.0f, pz = r.idir.z >= 0.0f;
    const uint32_t nx[2] = {px ? w2.x : w3.z, px ? w2.y : w3.w}, fx[2] = {px ? w3.z : w2.x, px ? w3.w : w2.y};
    const uint32_t ny[2] = {py ? w2.z : w4.x, py ? w2.w : w4.y}, fy[2] = {py ? w4.x : w2.z, py ? w4.y : w2.w};
    const uint32_t nz[2] = {pz ? w3.x : w4.z, pz ? w3.y : w4.w}, fz[2] = {pz ? w4.z : w3.x, pz ? w4.w : w3.y};
    // widen the interval by a few ulps so that rounding in the slab arithmetic can never
    // reject a box that the exact box test accepts
    const f32x2 widen = pack2(-1.0000010f, -1.0000010f), floor2 = pack2(-1e-30f, -1e-30f);
    uint32_t hmask = 0;
#pragma unroll
    for (int i = 6; i >= 0; i -= 2) {
        const int w = i >> 2, k = i & 3;
        const float2 txn = unpack2(fma2(byte_pair_alu(nx[w], k), ax2, bx2));
        const float2 tyn = unpack2(fma2(byte_pair_alu(ny[w], k), ay2, by2));
        const float2 tzn = unpack2(fma2(byte_pair(nz[w], k), az2, bz2));
        const float2 txf = unpack2(fma2(byte_pair_alu(fx[w], k), ax2, bx2));
        const float2 tyf = unpack2(fma2(byte_pair_alu(fy[w], k), ay2, by2));
        const float2 tzf = unpack2(fma2(byte_pair(fz[w], k), az2, bz2));
        // The slab interval with three-input integer min / max on the float bits (one
        // instruction each instead of two float ones).  Signed-integer order is float
        // order among non-negative floats and puts every negative float below them, so
        // tn, a maximum that includes tmin >= 0, is the float maximum exactly; tf is the
        // float minimum when it is non-negative and otherwise some negative candidate,
        // which rejects the box just as the float minimum does (tn >= 0) except within
        // 1e-30 of zero, where it can only accept a box more -- never reject one.
        auto tn = [&](float x, float y, float z) {
            return __int_as_float(__vimax3_s32(__float_as_int(x), __float_as_int(y), max(__float_as_int(z), __float_as_int(tmin))));
        };
        auto tf = [&](float x, float y, float z) {
            return __int_as_float(__vimin3_s32(__float_as_int(x), __float_as_int(y), min(__float_as_int(z), __float_as_int(tmax))));
        };
        // A child is hit when near <= far, that is when near - far, rounded down, has its
        // sign bit set (equal values give -0); the sign bits are shifted in.  A NaN gives the
        // canonical NaN, whose sign is clear: a ray with a NaN in its origin, its direction
        // or its t_min misses at the root instead of visiting every node.  (Taking the misses
        // from the sign of far - near let it visit all of them; both forms take the same
        // time: 2 M rays through 1.3 M triangles 366 us, the 16-scene batch 47.2 ms.)
        const f32x2 near = pack2(tn(txn.x, tyn.x, tzn.x), tn(txn.y, tyn.y, tzn.y));
        const f32x2 neg_far = fma2(pack2(tf(txf.x, tyf.x, tzf.x), tf(txf.y, tyf.y, tzf.y)), widen, floor2);
        const float2 gap = unpack2(add2_down(near, neg_far));
        hmask = __funnelshift_l(__float_as_uint(gap.y), hmask, 1);
        hmask = __funnelshift_l(__float_as_uint(gap.x), hmask, 1);
    }
    NodeHits h;
    // internal children hit, re-keyed slot -> slot ^ octant (three conditional swaps of
    // bit groups instead of a shift per child)
    uint32_t m = hmask & imask;
    if (r.flags & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (r.flags & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (r.flags & 4u) m = ((m & 0x0fu) << 4) | ((m >> 4) & 0x0fu);
    // leaf children hit: each hit bit widened to its child's three primitive bits
    uint32_t x = hmask;
    x = (x | (x << 8)) & 0x00f00fu;
    x = (x | (x << 4)) & 0x0c30c3u;
    x = (x | (x << 2)) & 0x249249u;
    h.child_base = w1.x;
    h.node_bits = m << 24 | imask;
    h.prim_base = w1.y;
    h.lmask = w1.z;
    h.prim_bits = x * 7u & w1.z;
    return h;
}

// Leaf primitive test against record `slot` of the leaf array; true when the primitive
// becomes the ray's hit (closest queries also need t < tbest, which is then updated).
// Closest-hit acceptance follows the reference: a triangle of a mesh is accepted when
// IntersectTriangle(t_min, t_best) succeeds and not (t > t_best || t <= 0)
// (triangle.cpp:211-225, bvh_aggregate.cpp:108-115; t < t_best already holds, and the
// record's second word tells mesh triangles from rectangle halves); rectangle halves skip
// the second check (rectangle.cpp:42-56); spheres use the inclusive range
// (sphere.cpp:116-127).  sphere(i, t) runs the test of sphere i, which needs the
// untransformed ray that the caller does not keep in registers.
template <class SphereTest>
FM_D bool test_prim(const float4* __restrict__ rec, const RayTrav& r, float tmin, float& tbest, Hit& hit, bool any,
                    SphereTest sphere)
{
    // all three records at once (a sphere's slot has them too), so the loads overlap
    const float4 a = __ldg(rec);
    const float4 b = __ldg(rec + 1);
    const float4 c = __ldg(rec + 2);
    const uint32_t tag = __float_as_uint(a.w);
    float t, b1 = 0.0f, b2 = 0.0f;
    if (tag & kSphereFlag) {
        if (!sphere((int)__float_as_uint(a.x), t)) return false;
    } else {
        if (!intersect_triangle(ray_axis(r), r.sx, r.sy, r.sz, r.no, a, b, c, tmin, tbest, t, b1, b2)) return false;
        if (!any && t <= 0.0f && b.w != 0.0f) return false;
    }
    hit.prim = (int)(tag & ~kSphereFlag);
    if (!any) {
        tbest = t;
        hit.b1 = b1;
        hit.b2 = b2;
    }
    return true;
}

// A per-thread traversal stack in local memory.
struct LocalStack {
    uint2 e[kTraversalStack];
    FM_D void put(int i, uint2 v) { e[i] = v; }
    FM_D uint2 get(int i) const { return e[i]; }
};

// A traversal stack whose K top entries are in shared memory (entry i of thread tid at
// top[i * stride], stride = the block size, so a warp's accesses are consecutive 8-byte
// words) and whose deeper entries are in local memory.
template <int K>
struct SharedTopStack {
    uint2* top;
    int stride;
    uint2 e[kTraversalStack - K];
    FM_D void put(int i, uint2 v)
    {
        if (i < K)
            top[i * stride] = v;
        else
            e[i - K] = v;
    }
    FM_D uint2 get(int i) const { return i < K ? top[i * stride] : e[i - K]; }
};

// The group a traversal starts with: a virtual parent whose only internal child, in slot
// 0, is the root (none for an empty tree).
FM_D uint2 root_group(int num_nodes, uint32_t oct)
{
    return num_nodes == 0 ? make_uint2(0u, 0u) : make_uint2(0u, (1u << (24 + oct)) | 1u);
}

// Takes the nearest pending child of `group` (which has one) off it and pushes what is
// left; returns the child's node index.  *overflow is set when the stack would overflow
// (the builder bounds the tree depth so that this cannot happen for trees it accepted).
template <class Stack>
FM_D uint32_t next_child(uint2& group, uint32_t oct, int& sp, Stack& stack, uint32_t* overflow)
{
    const uint32_t key = 31u - __clz(group.y) - 24u;
    group.y &= ~(1u << (24u + key));
    const uint32_t slot = key ^ oct;
    const uint32_t imask = group.y & 0xffu;
    const uint32_t child = group.x + __popc(imask & ((1u << slot) - 1u));
    if (group.y > 0x00ffffffu) {
        if (sp < kTraversalStack)
            stack.put(sp++, group);
        else if (overflow)
            atomicOr(overflow, 1u);
    }
    return child;
}

// Closest hit (any = false) or occlusion (any = true) query; hit.prim >= 0 on a hit.
// One ray per thread, for callers whose rays come one at a time (the megakernel); not
// inlined: a kernel that traces several kinds of rays holds one copy of the traversal
// loop, which keeps its code within the instruction caches.
static __device__ __noinline__ Hit trace_ray_any(const uint4* nodes, const float4* leaf, const SphereDev* spheres,
                                                 int num_nodes, f3 o, f3 d, float tmin, float tmax, bool any,
                                                 uint32_t* overflow)
{
    LocalStack stack;
    const RayTrav r = ray_trav(o, d);
    Hit hit{tmax, -1, 0.0f, 0.0f};
    uint2 group = root_group(num_nodes, ray_octant(r));
    int sp = 0;
    for (;;) {
        if (group.y <= 0x00ffffffu) {
            if (sp == 0) return hit;
            group = stack.get(--sp);
        }
        const uint32_t child = next_child(group, ray_octant(r), sp, stack, overflow);
        const NodeHits h = intersect_node(nodes + 5 * (size_t)child, r, tmin, hit.t);
        group = make_uint2(h.child_base, h.node_bits);
        for (uint32_t bits = h.prim_bits; bits; bits &= bits - 1u) {
            const uint32_t below = (bits & (0u - bits)) - 1u;
            const float4* rec = leaf + 3 * (size_t)(h.prim_base + __popc(h.lmask & below));
            auto sphere = [&](int i, float& t) {
                const SphereDev& s = spheres[i];
                return intersect_sphere(s.w2o, s.radius, o, d, tmin, hit.t, t);
            };
            if (test_prim(rec, r, tmin, hit.t, hit, any, sphere) && any) return hit;
        }
    }
}

template <bool ANY>
FM_D bool trace_ray(const DevScene& S, f3 o, f3 d, float tmin, float tmax, Hit& hit, uint32_t* overflow)
{
    hit = trace_ray_any(S.nodes, S.leaf, S.spheres, S.num_nodes, o, d, tmin, tmax, ANY, overflow);
    return hit.prim >= 0;
}

}  // namespace fm
