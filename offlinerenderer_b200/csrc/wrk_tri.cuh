// The ray-triangle test of the traversal kernels (trace.cu), shared with the
// Lambert shade (render.cu), which answers the shadow queries whose light triangle
// blocks the ray itself.
#pragma once
#include "wrk_internal.h"
#include "wrk_shading.cuh"

namespace wrk {

struct Ray {
    float ox, oy, oz, dx, dy, dz, tmin, tmax;
};

// Moller-Trumbore without the reciprocal: barycentric numerators are compared
// with det (sign-aware) and t is divided only for hits inside the triangle.  Each
// cross-product component is one product and one FMA, each dot product one product
// and two FMAs (correctly rounded intrinsics, in the CPU oracle's exact order).
__device__ __forceinline__ bool mt_rn(const Ray& r, float4 a, float4 b, float4 c, float& t) {
    float px = __fmaf_rn(r.dy, c.z, -__fmul_rn(r.dz, c.y));
    float py = __fmaf_rn(r.dz, c.x, -__fmul_rn(r.dx, c.z));
    float pz = __fmaf_rn(r.dx, c.y, -__fmul_rn(r.dy, c.x));
    float det = __fmaf_rn(b.x, px, __fmaf_rn(b.y, py, __fmul_rn(b.z, pz)));
    float sx = __fsub_rn(r.ox, a.x), sy = __fsub_rn(r.oy, a.y), sz = __fsub_rn(r.oz, a.z);
    float un = __fmaf_rn(sx, px, __fmaf_rn(sy, py, __fmul_rn(sz, pz)));
    float qx = __fmaf_rn(sy, b.z, -__fmul_rn(sz, b.y));
    float qy = __fmaf_rn(sz, b.x, -__fmul_rn(sx, b.z));
    float qz = __fmaf_rn(sx, b.y, -__fmul_rn(sy, b.x));
    float vn = __fmaf_rn(r.dx, qx, __fmaf_rn(r.dy, qy, __fmul_rn(r.dz, qz)));
    float uv = __fadd_rn(un, vn);
    bool inside = det > 0.0f ? (un >= 0.0f && vn >= 0.0f && uv <= det)
                             : (det < 0.0f && un <= 0.0f && vn <= 0.0f && uv >= det);
    if (!inside) return false;
    t = __fdiv_rn(__fmaf_rn(c.x, qx, __fmaf_rn(c.y, qy, __fmul_rn(c.z, qz))), det);
    return true;
}

// mt_rn for the two triangles of a pair record (kPairWords float4: the triangles at
// one leaf position and the next, component by component), the same operations on
// each half.  num / det: t's numerator and denominator where inside.
constexpr uint32_t kPairWords = 5;
__device__ __forceinline__ void mt_pair(const Ray& r, const float4* __restrict__ p, float2& num, float2& det, bool& in0,
                                        bool& in1) {
    const float4 p0 = __ldg(p), p1 = __ldg(p + 1), p2 = __ldg(p + 2), p3 = __ldg(p + 3), p4 = __ldg(p + 4);
    const f32x2 ax = pack2(p0.x, p0.y), ay = pack2(p0.z, p0.w), az = pack2(p1.x, p1.y), bx = pack2(p1.z, p1.w),
                by = pack2(p2.x, p2.y), bz = pack2(p2.z, p2.w), cx = pack2(p3.x, p3.y), cy = pack2(p3.z, p3.w),
                cz = pack2(p4.x, p4.y);
    const f32x2 dx = pack2(r.dx, r.dx), dy = pack2(r.dy, r.dy), dz = pack2(r.dz, r.dz);
    const f32x2 nx = pack2(-r.dx, -r.dx), ny = pack2(-r.dy, -r.dy), nz = pack2(-r.dz, -r.dz);
    // -(a * b) is exactly (-a) * b: the products below are the negated ones of mt_rn
    const f32x2 px = fma2(dy, cz, mul2(nz, cy)), py = fma2(dz, cx, mul2(nx, cz)), pz = fma2(dx, cy, mul2(ny, cx));
    const f32x2 d = fma2(bx, px, fma2(by, py, mul2(bz, pz)));
    // s = o - a; the records hold -v0
    const f32x2 sx = add2(pack2(r.ox, r.ox), ax), sy = add2(pack2(r.oy, r.oy), ay), sz = add2(pack2(r.oz, r.oz), az);
    const f32x2 un = fma2(sx, px, fma2(sy, py, mul2(sz, pz)));
    const f32x2 mone = pack2(-1.0f, -1.0f);
    const f32x2 tx = mul2(sx, mone), ty = mul2(sy, mone), tz = mul2(sz, mone);
    const f32x2 qx = fma2(sy, bz, mul2(tz, by)), qy = fma2(sz, bx, mul2(tx, bz)), qz = fma2(sx, by, mul2(ty, bx));
    const f32x2 vn = fma2(dx, qx, fma2(dy, qy, mul2(dz, qz)));
    const f32x2 uv = add2(un, vn);
    const f32x2 tn = fma2(cx, qx, fma2(cy, qy, mul2(cz, qz)));
    float u0, u1, v0, v1, w0, w1;
    unpack2(un, u0, u1);
    unpack2(vn, v0, v1);
    unpack2(uv, w0, w1);
    unpack2(d, det.x, det.y);
    unpack2(tn, num.x, num.y);
    auto inside = [](float dt, float u, float v, float w) {
        return dt > 0.0f ? (u >= 0.0f && v >= 0.0f && w <= dt) : (dt < 0.0f && u <= 0.0f && v <= 0.0f && w >= dt);
    };
    in0 = inside(det.x, u0, v0, w0);
    in1 = inside(det.y, u1, v1, w1);
}

// Does the ray hit the light triangle of light record `lr` (v0, v1, v2 in its first
// three float4s) within [tmin, tmax]?  The triangle is rebuilt as the BVH builder
// writes it (v0, v1 - v0, v2 - v0 with correctly rounded subtractions), so the
// answer is the one the traversal's triangle test gives for the same triangle.
__device__ __forceinline__ bool light_blocks(const float4* lr, const Ray& r) {
    const float4 l0 = __ldg(lr), l1 = __ldg(lr + 1), l2 = __ldg(lr + 2);
    const float4 a = make_float4(l0.x, l0.y, l0.z, 0.0f);
    const float4 b = make_float4(__fsub_rn(l1.x, l0.x), __fsub_rn(l1.y, l0.y), __fsub_rn(l1.z, l0.z), 0.0f);
    const float4 c = make_float4(__fsub_rn(l2.x, l0.x), __fsub_rn(l2.y, l0.y), __fsub_rn(l2.z, l0.z), 0.0f);
    float th;
    return mt_rn(r, a, b, c, th) && th >= r.tmin && th <= r.tmax;
}

}  // namespace wrk
