// Ray/primitive intersection with the reference's exact float arithmetic.
//
// Closest-hit primitive IDs must match the reference's built-in BVH bit for bit, so the
// triangle test performs the same IEEE float operations in the same order as
// triangle_func::IntersectTriangle (src/engine/src/geometry/triangle.cpp:25-94), with
// every multiply and add written as an explicitly rounded intrinsic so that the compiler
// cannot contract them into FMAs.  The double-precision fallback of triangle.cpp:61-66
// is reproduced with explicitly rounded double operations.
//
// The main-axis choice reproduces triangle.cpp:13-18 as the reference compiles: the
// unqualified `abs` there binds to the C library's int abs(int), so each direction
// component is truncated toward zero before the comparison (so the test almost always
// permutes z to the main axis).  The oracle's known-answer test pins this binding.
#pragma once
#include "fm_common.cuh"

namespace fm {

// Two floats processed by one packed instruction (sm_100's f32x2 arithmetic).  Each half
// is rounded as the scalar IEEE operation is, so results equal the scalar code's bit for
// bit in half the issue slots.  There is no packed multiply here: ptxas contracts
// mul.rn.f32x2 followed by add.rn.f32x2 into one multiply-add, unlike their scalar forms.
typedef unsigned long long f32x2;
FM_D f32x2 pack2(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
FM_D float2 unpack2(f32x2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
FM_D f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
FM_D f32x2 add2_down(f32x2 a, f32x2 b)   // rounded towards minus infinity
{
    f32x2 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
FM_D f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Per-ray constants of the watertight test: the main axis kz (the permutation is
// (kz+1, kz+2, kz) mod 3) and the shear.
struct RayPre {
    int kz;
    float sx, sy, sz;
};

FM_D int trunc_abs(float v)
{
    // (int)v then abs(): float -> int conversion truncates toward zero.
    const int i = __float2int_rz(v);
    return i < 0 ? -i : i;
}

FM_D RayPre ray_pre(f3 d)
{
    RayPre p;
    const int a0 = trunc_abs(d.x), a1 = trunc_abs(d.y), a2 = trunc_abs(d.z);
    int az;
    if (a0 > a1 && a0 > a2)
        az = 0;
    else
        az = a1 > a2 ? 1 : 2;
    // A main-axis component of zero (or so small that 1/dz overflows) makes the shear
    // infinite and every edge function NaN; the reference then reports NaN hits.  Its
    // double build practically never draws such a ray, but float sampling does (a
    // cosine-hemisphere sample at an axis-aligned wall has d.z == 0 exactly about once
    // in 2^24 draws), so those rays use the axis of largest magnitude instead.  Rays
    // with |dz| >= 1e-30 keep the reference's choice and its results bit for bit.
    if (!(fabsf(comp(d, az)) >= 1e-30f)) {
        const float m0 = fabsf(d.x), m1 = fabsf(d.y), m2 = fabsf(d.z);
        az = (m0 >= m1 && m0 >= m2) ? 0 : (m1 >= m2 ? 1 : 2);
    }
    const int ax = (az + 1) % 3;
    const int ay = (ax + 1) % 3;
    p.kz = az;
    const float dx = comp(d, ax), dy = comp(d, ay), dz = comp(d, az);
    p.sx = __fdiv_rn(-dx, dz);
    p.sy = __fdiv_rn(-dy, dz);
    p.sz = __fdiv_rn(1.0f, dz);
    return p;
}

FM_D float edge_double(float ax, float ay, float bx, float by)
{
    // (real)((double)ax * (double)by - (double)ay * (double)bx)
    return __double2float_rn(__dsub_rn(__dmul_rn((double)ax, (double)by), __dmul_rn((double)ay, (double)bx)));
}

// triangle_func::IntersectTriangle.  Returns true on a hit with t in (tmin, tmax).  The
// reference's rejection test (t <= tmin || t >= tmax) lets a NaN t through; here a NaN
// t is rejected as well (it arises only from degenerate input, never on a ray the
// reference handles with finite arithmetic).
//
// no is the negated ray origin (x + (-o) is x - o exactly); a, b and c hold the corners in
// xyz.  x and y take the same steps, so their additions run as packed pairs: 15 instead
// of 21 instructions for the three corners.  The permutation is the identity
// whenever z is the main axis, which the truncating main-axis choice makes it for almost
// every ray; other axes take a branch that swaps components.
FM_D bool intersect_triangle(int kz, float sx, float sy, float sz, f3 no, float4 a, float4 b, float4 c, float tmin,
                             float tmax, float& t_out, float& b1, float& b2)
{
    // translate
    const f32x2 noxy = pack2(no.x, no.y);
    f32x2 q0 = add2(pack2(a.x, a.y), noxy), q1 = add2(pack2(b.x, b.y), noxy), q2 = add2(pack2(c.x, c.y), noxy);
    float p0z = __fadd_rn(a.z, no.z), p1z = __fadd_rn(b.z, no.z), p2z = __fadd_rn(c.z, no.z);
    // permute
    if (kz != 2) {
        auto perm = [&](f32x2& xy, float& z) {
            const float2 v = unpack2(xy);
            xy = kz == 0 ? pack2(v.y, z) : pack2(z, v.x);
            z = kz == 0 ? v.x : v.y;
        };
        perm(q0, p0z);
        perm(q1, p1z);
        perm(q2, p2z);
    }
    // shear
    const float2 p0 = unpack2(add2(q0, pack2(__fmul_rn(sx, p0z), __fmul_rn(sy, p0z))));
    const float2 p1 = unpack2(add2(q1, pack2(__fmul_rn(sx, p1z), __fmul_rn(sy, p1z))));
    const float2 p2 = unpack2(add2(q2, pack2(__fmul_rn(sx, p2z), __fmul_rn(sy, p2z))));
    // edge functions
    float e0 = __fsub_rn(__fmul_rn(p1.x, p2.y), __fmul_rn(p1.y, p2.x));
    float e1 = __fsub_rn(__fmul_rn(p2.x, p0.y), __fmul_rn(p2.y, p0.x));
    float e2 = __fsub_rn(__fmul_rn(p0.x, p1.y), __fmul_rn(p0.y, p1.x));
    if (e0 == 0.0f || e1 == 0.0f || e2 == 0.0f) {
        e0 = edge_double(p1.x, p1.y, p2.x, p2.y);
        e1 = edge_double(p2.x, p2.y, p0.x, p0.y);
        e2 = edge_double(p0.x, p0.y, p1.x, p1.y);
    }
    if ((e0 < 0 || e1 < 0 || e2 < 0) && (e0 > 0 || e1 > 0 || e2 > 0)) return false;
    const float det = __fadd_rn(__fadd_rn(e0, e1), e2);
    if (det == 0) return false;
    p0z = __fmul_rn(p0z, sz);
    p1z = __fmul_rn(p1z, sz);
    p2z = __fmul_rn(p2z, sz);
    const float inv_det = __fdiv_rn(1.0f, det);
    const float t = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(e0, p0z), __fmul_rn(e1, p1z)), __fmul_rn(e2, p2z)), inv_det);
    if (t <= tmin || t >= tmax || t != t) return false;
    t_out = t;
    b1 = __fmul_rn(e1, inv_det);
    b2 = __fmul_rn(e2, inv_det);
    return true;
}

// Sphere::IntersectSphere (geometry/sphere.cpp:91-129, GetCoef :206-212): the ray is
// taken to object space (not renormalized, so t is shared), the quadratic is solved
// without the robust form, and the nearer root inside the inclusive range [tmin, tmax]
// is returned.  Every operation is explicitly rounded in the reference's order
// (SquareSum and glm::dot left to right, b*b - (4a)*c, 0.5/a), so no multiply-add is
// contracted and the result equals the reference's float build bit for bit whenever the
// object-space ray does (always for translation-only transforms, whose world-to-object
// step is one rounded subtraction per origin component and exact for the direction).
FM_D bool intersect_sphere(const Xf& world_to_object, float radius, f3 o, f3 d, float tmin, float tmax,
                           float& t_out)
{
    const f3 ol = xf_point(world_to_object, o);
    const f3 dl = xf_vec(world_to_object, d);
    const float a = __fadd_rn(__fadd_rn(__fmul_rn(dl.x, dl.x), __fmul_rn(dl.y, dl.y)), __fmul_rn(dl.z, dl.z));
    const float b =
        __fmul_rn(2.0f, __fadd_rn(__fadd_rn(__fmul_rn(dl.x, ol.x), __fmul_rn(dl.y, ol.y)), __fmul_rn(dl.z, ol.z)));
    const float c = __fsub_rn(__fadd_rn(__fadd_rn(__fmul_rn(ol.x, ol.x), __fmul_rn(ol.y, ol.y)), __fmul_rn(ol.z, ol.z)),
                              __fmul_rn(radius, radius));
    float delta = __fsub_rn(__fmul_rn(b, b), __fmul_rn(__fmul_rn(4.0f, a), c));
    if (delta < 0) return false;
    delta = __fsqrt_rn(delta);
    const float inv2a = __fdiv_rn(0.5f, a);
    const float t0 = __fmul_rn(__fsub_rn(-b, delta), inv2a);
    const float t1 = __fmul_rn(__fadd_rn(-b, delta), inv2a);
    if (t0 >= tmin && t0 <= tmax) {
        t_out = t0;
        return true;
    }
    if (t1 >= tmin && t1 <= tmax) {
        t_out = t1;
        return true;
    }
    return false;
}

}  // namespace fm
