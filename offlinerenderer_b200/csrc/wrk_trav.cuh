// Device code of the 8-wide BVH traversal, shared by the wavefront trace kernels and ray
// queries (trace.cu) and the one-launch renderer of small images (render.cu).
//
// Per node: five 16-byte loads (__ldg, read-only path), eight quantized slab tests
// decoded with one byte permute per plane and one packed FMA per near / far plane pair.
// Internal-child hits go into an 8-bit mask permuted by the ray octant so the
// lowest set bit is the child nearest the ray's entry corner; leaf-child hits set
// bits of a triangle mask.  Pending node groups
// (child base + remaining hit bits + internal mask) go on a short stack held in
// shared memory, spilling to a bounded local array; overflow raises an error bit
// and ends the ray instead of corrupting memory.
//
// The triangle test is Moller-Trumbore in packed FP32 pairs (two triangles a test), on
// each half the same sequence of correctly rounded operations as the CPU oracle's.
#pragma once
#include "wrk_internal.h"
#include "wrk_shading.cuh"
#include "wrk_tri.cuh"

namespace wrk {

constexpr int kTraceBlock = 128;
// Stack entries per lane in shared memory (the rest, rarely used, in local memory).
constexpr int kStackSmem = 8;
constexpr int kStackLocal = 48 - kStackSmem;
constexpr uint32_t kMaxVisits = 1u << 16;
// Byte k of w as the float 2^15 + b, exactly, without an int->float conversion:
// one byte permute builds the bits 0x4700bb00 (exponent 2^15, b in mantissa bits
// 8-15).  The 2^15 bias is folded into the per-node plane offset (see
// intersect_node).
__device__ __forceinline__ float qbias(uint32_t w, uint32_t k) {
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7504u | (k << 4)));
}

// Intersects the 8 children of a node; returns internal hits (permuted by octant)
// and the triangle mask relative to triBase.
//
// The node test is issue- and ALU-bound (byte permutes and min / max run at half
// rate), so an axis' near and far planes share one packed FMA, and a child's outcome
// is the sign of one FMA shifted into the hit mask.  With the refill below, 1M rays
// against a 676k-triangle scene (closest hit + occlusion): 803 -> 753 us.
__device__ __forceinline__ void intersect_node(const uint4* __restrict__ nodes, uint32_t idx, float ox, float oy,
                                               float oz, float ix, float iy, float iz, uint32_t oct_inv, float tmin,
                                               float tfar_max, uint32_t& childBase, uint32_t& triBase,
                                               uint32_t& hits, uint32_t& imask, uint32_t& tmask) {
    const uint4* n = nodes + 5 * (size_t)idx;
    uint4 n0 = __ldg(n), n1 = __ldg(n + 1), n2 = __ldg(n + 2), n3 = __ldg(n + 3), n4 = __ldg(n + 4);
    float px = __uint_as_float(n0.x), py = __uint_as_float(n0.y), pz = __uint_as_float(n0.z);
    float sx = __uint_as_float((n0.w & 0xffu) << 23) * ix;
    float sy = __uint_as_float(((n0.w >> 8) & 0xffu) << 23) * iy;
    float sz = __uint_as_float(((n0.w >> 16) & 0xffu) << 23) * iz;
    float ax = (px - ox) * ix, ay = (py - oy) * iy, az = (pz - oz) * iz;
    // plane t = q*s + a = (2^15 + q)*s + (a - 2^15*s).  The biased offsets are
    // rounded down for near planes and up for far planes, so their rounding only
    // grows the slab (by at most ~1/256 of a quantization step); the plane FMAs
    // round to nearest (2^-24 of t), which the 2^-22 slack of the test below covers:
    // a child box the ray crosses is never rejected.
    const f32x2 sx2 = pack2(sx, sx), sy2 = pack2(sy, sy), sz2 = pack2(sz, sz);
    const f32x2 ax2 = pack2(__fmaf_rd(-32768.0f, sx, ax), __fmaf_ru(-32768.0f, sx, ax));
    const f32x2 ay2 = pack2(__fmaf_rd(-32768.0f, sy, ay), __fmaf_ru(-32768.0f, sy, ay));
    const f32x2 az2 = pack2(__fmaf_rd(-32768.0f, sz, az), __fmaf_ru(-32768.0f, sz, az));
    imask = n0.w >> 24;
    childBase = n1.x;
    triBase = n1.y;
    // near/far plane words per axis: dir >= 0 -> near = lo, far = hi
    uint32_t xn0 = ix >= 0.0f ? n2.x : n3.z, xn1 = ix >= 0.0f ? n2.y : n3.w;
    uint32_t xf0 = ix >= 0.0f ? n3.z : n2.x, xf1 = ix >= 0.0f ? n3.w : n2.y;
    uint32_t yn0 = iy >= 0.0f ? n2.z : n4.x, yn1 = iy >= 0.0f ? n2.w : n4.y;
    uint32_t yf0 = iy >= 0.0f ? n4.x : n2.z, yf1 = iy >= 0.0f ? n4.y : n2.w;
    uint32_t zn0 = iz >= 0.0f ? n3.x : n4.z, zn1 = iz >= 0.0f ? n3.y : n4.w;
    uint32_t zf0 = iz >= 0.0f ? n4.z : n3.x, zf1 = iz >= 0.0f ? n4.w : n3.y;
    const float tfar_lim = tfar_max * 1.00000024f;
    uint32_t hm = 0;  // children whose slab the ray crosses, by slot
#pragma unroll
    for (int s = 7; s >= 0; --s) {
        const uint32_t k = s & 3;
        uint32_t xn = s < 4 ? xn0 : xn1, xf = s < 4 ? xf0 : xf1;
        uint32_t yn = s < 4 ? yn0 : yn1, yf = s < 4 ? yf0 : yf1;
        uint32_t zn = s < 4 ? zn0 : zn1, zf = s < 4 ? zf0 : zf1;
        float t0x, t1x, t0y, t1y, t0z, t1z;
        unpack2(fma2(pack2(qbias(xn, k), qbias(xf, k)), sx2, ax2), t0x, t1x);
        unpack2(fma2(pack2(qbias(yn, k), qbias(yf, k)), sy2, ay2), t0y, t1y);
        unpack2(fma2(pack2(qbias(zn, k), qbias(zf, k)), sz2, az2), t0z, t1z);
        // Three-input integer max / min on the float bit patterns.  Non-negative
        // floats order like their bit patterns; negative ones order reversed, which
        // only moves tn down and tf up (a larger slab, never a smaller one), and a
        // negative tf still fails against tn >= tmin >= 0.
        float tn = __int_as_float(__vimax3_s32(__float_as_int(t0x), __float_as_int(t0y),
                                               max(__float_as_int(t0z), __float_as_int(tmin))));
        float tf = __int_as_float(__vimin3_s32(__float_as_int(t1x), __float_as_int(t1y),
                                               min(__float_as_int(t1z), __float_as_int(tfar_lim))));
        // crossed when tn - tf * (1 + 2^-22) <= 0: the sign of one FMA (rounded down, so
        // that an exact zero is -0; a NaN, from a NaN ray, has its sign clear: missed)
        hm = __funnelshift_l(__float_as_uint(__fmaf_rd(tf, -1.00000024f, tn)), hm, 1);
    }
    // internal hits, moved from slot s to bit s ^ oct_inv by three conditional swaps
    uint32_t ih = hm & imask;
    if (oct_inv & 1u) ih = ((ih & 0x55u) << 1) | ((ih >> 1) & 0x55u);
    if (oct_inv & 2u) ih = ((ih & 0x33u) << 2) | ((ih >> 2) & 0x33u);
    if (oct_inv & 4u) ih = ((ih & 0x0Fu) << 4) | ((ih >> 4) & 0x0Fu);
    hits = ih;
    // leaf hits: each adds its run of cnt triangles starting at bit off
    uint32_t lh = hm & ~imask;
    tmask = 0;
    while (lh) {
        const uint32_t j = __ffs(lh) - 1;
        lh &= lh - 1;
        const uint32_t meta = ((j < 4 ? n1.z : n1.w) >> (8 * (j & 3u))) & 0xffu;
        const uint32_t cnt = (meta >> 5) + 1u, off = meta & 31u;
        tmask |= ((1u << cnt) - 1u) << off;
    }
}

// The scene fields traversal needs (a DevScene has them too).
struct TraceGeom {
    const uint4* nodes;
    const float4* tris;
    const float4* pairs;
    uint32_t numNodes, numTris;
};

// Per-lane traversal state, kept in registers across the persistent loop's rounds: every
// word of it counts (an extension kernel that spills runs several percent slower).
constexpr uint32_t kOctShift = 8, kVisitShift = 11;
struct Trav {
    float ox, oy, oz;
    float ix, iy, iz;
    uint32_t gBase;
    uint32_t gBits;  // node group: child hit bits (bits 0-7, octant order) | internal-child mask << 8
    uint32_t state;  // stack entries (bits 0-7) | ray octant, inverted (8-10) | nodes visited << 11
    float tBest;
    // Leaf position (index into the BVH triangle records) of the best hit, kNoHit
    // while there is none; the hit's primitive and material are read from that
    // record when the ray is done, so they take no registers during traversal.
    uint32_t lBest;
};

__device__ __forceinline__ uint32_t record_prim(const float4* tris, uint32_t l) {
    return l == kNoHit ? kNoHit : __float_as_uint(__ldg(tris + 3 * (size_t)l).w);
}
__device__ __forceinline__ uint32_t record_material(const float4* tris, uint32_t l) {
    return l == kNoHit ? 0u : __float_as_uint(__ldg(tris + 3 * (size_t)l + 1).w);
}

__device__ __forceinline__ void trav_init(Trav& t, float4* sdir, const Ray& r) {
    t.ox = r.ox;
    t.oy = r.oy;
    t.oz = r.oz;
    sdir[threadIdx.x] = make_float4(r.dx, r.dy, r.dz, r.tmin);
    // Direction components below 2^-80 in magnitude are replaced by +-2^-80 for
    // the slab tests only (the triangle test uses the true direction), so inverse
    // directions and plane distances stay finite and never NaN.
    const float ooeps = 8.27180613e-25f;
    t.ix = 1.0f / (fabsf(r.dx) < ooeps ? copysignf(ooeps, r.dx) : r.dx);
    t.iy = 1.0f / (fabsf(r.dy) < ooeps ? copysignf(ooeps, r.dy) : r.dy);
    t.iz = 1.0f / (fabsf(r.dz) < ooeps ? copysignf(ooeps, r.dz) : r.dz);
    uint32_t oct = (r.dx < 0.0f ? 1u : 0u) | (r.dy < 0.0f ? 2u : 0u) | (r.dz < 0.0f ? 4u : 0u);
    const uint32_t octInv = oct ^ 7u;  // slot of the child nearest the entry corner -> bit 0
    t.state = octInv << kOctShift;
    // the root is a one-child node group
    t.gBase = 0;
    t.gBits = (1u << octInv) | (1u << 8);
    t.tBest = r.tmax;
    t.lBest = kNoHit;
}

// One traversal step: descend into the next child of the current node group
// (pushing the group's remainder), test the triangles that node exposes, and pop
// when the group is used up.  Returns true when the ray is finished.  Closest hit
// keeps ties in t with the lower primitive index; any hit stops at the first hit.
// kTmin0: every ray's tmin is at least 0, so the node test clamps at 0 (the triangle
// test always applies the ray's own); otherwise at the ray's tmin.
template <bool kAnyHit, bool kTmin0, class Geom>
__device__ __forceinline__ bool trav_step(const Geom& s, Trav& t, const float4* sdir, uint2* sstack, uint2* lstack,
                                          uint32_t* errFlag) {
    const int tid = threadIdx.x;
    t.state += 1u << kVisitShift;
    if (t.state >> kVisitShift > kMaxVisits) {  // a malformed tree must not spin forever
        atomicOr(errFlag, kErrBadIndex);
        return true;
    }
    uint32_t tBase = 0, tMask = 0;  // the triangles the node exposes
    if (t.gBits & 0xffu) {
        const uint32_t octInv = (t.state >> kOctShift) & 7u;
        uint32_t pos = __ffs(t.gBits) - 1;  // the lowest set bit is a hit bit
        t.gBits &= t.gBits - 1;
        uint32_t slot = pos ^ octInv;
        uint32_t child = t.gBase + __popc(t.gBits & (((1u << slot) - 1u) << 8));
        if (t.gBits & 0xffu) {
            uint2 e = make_uint2(t.gBase, t.gBits);
            const int sp = t.state & 0xffu;
            if (sp < kStackSmem) sstack[sp * kTraceBlock + tid] = e;
            else if (sp < kStackSmem + kStackLocal) lstack[sp - kStackSmem] = e;
            else {
                atomicOr(errFlag, kErrStackOverflow);
                return true;
            }
            ++t.state;
        }
        if (child >= s.numNodes) {
            atomicOr(errFlag, kErrBadIndex);
            return true;
        }
        uint32_t hits, imask;
        intersect_node(s.nodes, child, t.ox, t.oy, t.oz, t.ix, t.iy, t.iz, octInv, kTmin0 ? 0.0f : sdir[tid].w, t.tBest,
                       t.gBase, tBase, hits, imask, tMask);
        t.gBits = hits | (imask << 8);
        if (tMask && tBase + (31u - __clz(tMask)) >= s.numTris) {
            atomicOr(errFlag, kErrBadIndex);
            return true;
        }
    }
    // A leaf's triangles occupy a handful of lanes while the others wait, so two are
    // tested at a time (mt_pair), and the ray's direction, which only this part reads,
    // stays in shared memory: 64 registers without spills, where one triangle at a time
    // and the direction in registers took 58.  Showcase extension stage 34.0 -> 32.8 ms,
    // 1M-ray queries 753 -> 704 us.
    if (tMask) {
        const float4 dt = sdir[tid];
        const Ray r{t.ox, t.oy, t.oz, dt.x, dt.y, dt.z, dt.w, 0.0f};
        while (tMask) {
            // the lowest pending triangle and, when it is pending too, the next one, in one
            // packed test
            const uint32_t j = __ffs(tMask) - 1;
            const bool two = (tMask >> j) & 2u;
            tMask &= ~(3u << j);
            uint32_t l = tBase + j;
            float2 num, det;
            bool in0, in1;
            mt_pair(r, s.pairs + kPairWords * (size_t)l, num, det, in0, in1);
            in1 = in1 && two;
            if (!in0) {
                if (!in1) continue;
                ++l;
            }
            // both inside (a shared edge, coincident triangles): the first, then the second
            bool again = in0 && in1;
            float n = in0 ? num.x : num.y, d = in0 ? det.x : det.y;
            while (true) {
                const float th = __fdiv_rn(n, d);
                // closest hit: tBest <= tmax, so the update test below implies th <= tmax;
                // any hit: tBest is tmax until the first hit, which ends the ray
                if (th >= r.tmin && (!kAnyHit || th <= t.tBest)) {
                    if (kAnyHit) {
                        t.tBest = th;
                        t.lBest = l;
                        return true;
                    }
                    if (th < t.tBest || (th == t.tBest && record_prim(s.tris, l) < record_prim(s.tris, t.lBest))) {
                        t.tBest = th;
                        t.lBest = l;
                    }
                }
                if (!again) break;
                again = false;
                ++l;
                n = num.y;
                d = det.y;
            }
        }
    }
    if (!(t.gBits & 0xffu)) {
        const int sp = (int)(t.state & 0xffu) - 1;
        if (sp < 0) return true;
        --t.state;
        uint2 e = sp < kStackSmem ? sstack[sp * kTraceBlock + tid] : lstack[sp - kStackSmem];
        t.gBase = e.x;
        t.gBits = e.y;
    }
    return false;
}

// Adds a miss's environment term and accumulates the path into its request's sums
// (__miss__trace + the raygen miss branch, trace.cu:143-148).
__device__ __forceinline__ void miss_accumulate(const DevScene& sc, const Frame& f, float4 th, float4 rd, float3 dir) {
    float3 e = make_float3(sc.env[0], sc.env[1], sc.env[2]);
    if ((f.flags & WRK_FLAG_ENV_MAP) && sc.envMap) e = env_lookup(sc.envMap, sc.envW, sc.envH, dir);
    float3 L = make_float3(rd.x + th.x * e.x, rd.y + th.y * e.y, rd.z + th.z * e.z);
    L = clamp_fireflies(L, f.fireflyClamp);
    atomicAdd(f.accum + __float_as_uint(rd.w), make_float4(L.x, L.y, L.z, 0.0f));
}

}  // namespace wrk
