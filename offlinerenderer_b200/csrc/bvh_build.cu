// GPU BVH builder: binned-SAH binary tree, collapsed into an 8-wide BVH with
// quantized (compressed) child boxes.  Replaces optixAccelBuild
// (libWR/src/internal/scene.cpp:493-550 in trianglestrip/OfflineRenderer).
//
// Binary build, level by level over all open tasks at once:
//   bin     -- every primitive adds its AABB to its task's 16 bins on each axis
//              (atomics on order-preserving integer encodings of floats, merged per
//              block and task in shared memory)
//   split   -- one warp per task scans the bins for the lowest SAH cost of the 3x15
//              candidate planes (object median when all centroids share a bin);
//              allocates the two children; children of <= kSmallTask primitives go to
//              the small list
//   flags + exclusive scan + scatter -- stable partition of each task's range,
//              accumulating child boxes and centroid bounds with atomics.
// Small tasks are finished by a half-warp each with sorted SAH sweeps.
//
// Collapse: top-down, eight lanes per 8-wide node.  The binary child with the
// largest surface area is opened until 8 children; children go to slots by
// corner (octant) so traversal can visit them front-to-back by XOR with the ray's
// octant; child boxes are quantized to 8 bits against the node box, widened by one
// quantization step so decoding never shrinks a box.  Leaves' triangles are copied
// into leaf order as (v0|prim, v1-v0|material, v2-v0) records.
#include <cub/cub.cuh>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <mutex>

#include "wrk_internal.h"

namespace wrk {
namespace {

constexpr int kBins = 16;
constexpr uint32_t kSmallTask = 16;
constexpr uint32_t kMaxLeaf = 3;
// BVH levels (and collapse depths) enqueued between two host reads of the counts.
constexpr int kLevelsPerSync = 4;
constexpr uint32_t kMaxLevels = 256;

__host__ __device__ __forceinline__ uint32_t f2o(float f) {
#ifdef __CUDA_ARCH__
    uint32_t u = __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
#endif
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

struct alignas(16) BNode {
    float lo[3];
    uint32_t left;  // internal: left child (right = left+1); leaf: first primitive position
    float hi[3];
    uint32_t count;  // 0 = internal
};
struct OBox {
    uint32_t lo[3], hi[3];
};  // order-encoded floats, for atomic min/max
struct Task {
    uint32_t node, begin, end, pad;
};
struct alignas(16) Bin {
    uint32_t cnt;
    uint32_t lo[3], hi[3];
    uint32_t pad;
};
struct Split {
    int axis, bin;
    uint32_t nLeft;
    int leftTask, rightTask;  // >= 0 next-level task id, -1 prims finished
    uint32_t leftNode;
    uint32_t pad[2];
};
struct SmallTask {
    uint32_t node, begin, end, pad;
};
// cur: open tasks of the level being built (set on the device from nextTasks at the
// start of each level, so the host need not read it back between levels).
struct BuildCtr {
    uint32_t nodes, nextTasks, small, cur;
};
struct CollapseCtr {
    uint32_t nodes, tris, next, maxDepth, cur;
};

__device__ __forceinline__ void obox_empty(OBox& b) {
    for (int k = 0; k < 3; ++k) { b.lo[k] = f2o(FLT_MAX); b.hi[k] = f2o(-FLT_MAX); }
}

__global__ void k_prim_bounds(const float* __restrict__ vtx, const uint32_t* __restrict__ idx, uint32_t n,
                              float4* __restrict__ blo, float4* __restrict__ bhi, OBox* rootBox, OBox* rootCen) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    float c[3] = {0, 0, 0};
    bool valid = i < n;
    if (valid) {
        for (int v = 0; v < 3; ++v) {
            uint32_t k = idx[3 * i + v];
            for (int a = 0; a < 3; ++a) {
                float x = vtx[3 * k + a];
                lo[a] = fminf(lo[a], x);
                hi[a] = fmaxf(hi[a], x);
            }
        }
        blo[i] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        bhi[i] = make_float4(hi[0], hi[1], hi[2], 0.0f);
        for (int a = 0; a < 3; ++a) c[a] = 0.5f * (lo[a] + hi[a]);
    }
    // block-reduce to a few atomics
    typedef cub::BlockReduce<float, 256> BR;
    __shared__ typename BR::TempStorage tmp;
    for (int a = 0; a < 3; ++a) {
        float m = BR(tmp).Reduce(lo[a], cub::Min());
        __syncthreads();
        float M = BR(tmp).Reduce(hi[a], cub::Max());
        __syncthreads();
        float cm = BR(tmp).Reduce(valid ? c[a] : FLT_MAX, cub::Min());
        __syncthreads();
        float cM = BR(tmp).Reduce(valid ? c[a] : -FLT_MAX, cub::Max());
        __syncthreads();
        if (threadIdx.x == 0) {
            atomicMin(&rootBox->lo[a], f2o(m));
            atomicMax(&rootBox->hi[a], f2o(M));
            atomicMin(&rootCen->lo[a], f2o(cm));
            atomicMax(&rootCen->hi[a], f2o(cM));
        }
    }
}

// One thread, at the start of a level: the tasks the last level opened become this
// level's (the device keeps the count; the host reads it only every few levels).
__global__ void k_level_begin(BuildCtr* ctr) {
    ctr->cur = ctr->nextTasks;
    ctr->nextTasks = 0;
}

// The empty bin (32 bytes as two words: cnt, lo | hi, pad).
__device__ __forceinline__ void clear_bin(Bin* b) {
    const uint32_t lo = f2o(FLT_MAX), hi = f2o(-FLT_MAX);
    uint4* w = reinterpret_cast<uint4*>(b);
    w[0] = make_uint4(0u, lo, lo, lo);
    w[1] = make_uint4(hi, hi, hi, 0u);
}
// All bins, once per build; k_split empties the ones it has read.
__global__ void k_init_bins(Bin* bins, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) clear_bin(bins + i);
}
__global__ void k_iota(uint32_t* ref, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) ref[i] = i;
}

__device__ __forceinline__ int bin_of(float c, float lo, float ext) {
    if (!(ext > 0.0f)) return 0;
    int b = (int)((c - lo) * ((float)kBins / ext));
    return min(kBins - 1, max(0, b));
}

// A block's primitives occupy consecutive positions and a task's primitives one
// contiguous range, so a block meets a few tasks one after the other: its segments.  The
// first maxSeg of them are merged into shared-memory copies of the tasks' bins / child
// boxes, and each touched field takes one global atomic per block instead of one per
// primitive (near the root every primitive of the scene would otherwise hit the same few
// addresses).  Merging only blocks that lie in one task left the deep levels to atomics
// per primitive, and a warp's lanes to conflicts on one address: k_bin 1133 -> 655 us and
// k_scatter 941 -> 519 us per 676k-triangle build.
// min / max / add give the same result in any order, so the tree does not change.
//
// Returns this thread's segment; segTask[k] = the task of segment k < maxSeg (-1:
// finished primitives), *numSeg = segments.  All 256 threads call it.
__device__ __forceinline__ uint32_t block_segment(uint32_t n, const int* __restrict__ taskOf, uint32_t maxSeg, int* segTask,
                                                  uint32_t* numSeg) {
    __shared__ uint32_t warpStarts[8];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const int t = i < n ? taskOf[i] : -1;
    const bool start = threadIdx.x == 0 || (i < n && taskOf[i - 1] != t);
    const uint32_t m = __ballot_sync(0xffffffffu, start);
    if (lane == 0) warpStarts[warp] = __popc(m);
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (uint32_t w = 0; w < 8; ++w) {
        if (w < warp) before += warpStarts[w];
        total += warpStarts[w];
    }
    const uint32_t seg = before + __popc(m & (0xffffffffu >> (31u - lane))) - 1u;
    if (start && seg < maxSeg) segTask[seg] = t;
    *numSeg = min(total, maxSeg);
    return seg;
}

constexpr uint32_t kBinSegments = 8, kBoxSegments = 16;

__global__ void __launch_bounds__(256) k_bin(uint32_t n, const uint32_t* __restrict__ ref, const int* __restrict__ taskOf,
                                             const OBox* __restrict__ tcen, const float4* __restrict__ blo,
                                             const float4* __restrict__ bhi, Bin* bins) {
    __shared__ uint32_t sCnt[kBinSegments * 3 * kBins], sLo[kBinSegments * 3 * kBins][3], sHi[kBinSegments * 3 * kBins][3];
    __shared__ int segTask[kBinSegments];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t numSeg;
    const uint32_t seg = block_segment(n, taskOf, kBinSegments, segTask, &numSeg);
    for (uint32_t k = threadIdx.x; k < numSeg * 3 * kBins; k += blockDim.x) {
        sCnt[k] = 0;
        for (int c = 0; c < 3; ++c) { sLo[k][c] = 0xffffffffu; sHi[k][c] = 0u; }
    }
    __syncthreads();
    const int t = i < n ? taskOf[i] : -1;
    const uint32_t any = __ballot_sync(0xffffffffu, t >= 0);
    if (t >= 0) {
        const uint32_t p = ref[i];
        const float4 l = blo[p], h = bhi[p];
        const float lo[3] = {l.x, l.y, l.z}, hi[3] = {h.x, h.y, h.z};
        const OBox cb = tcen[t];
        const bool merged = seg < kBinSegments;
        uint32_t ol[3], oh[3];
        for (int c = 0; c < 3; ++c) { ol[c] = f2o(lo[c]); oh[c] = f2o(hi[c]); }
        for (int a = 0; a < 3; ++a) {
            const float cl = o2f(cb.lo[a]), ch = o2f(cb.hi[a]);
            const uint32_t b = (uint32_t)a * kBins + bin_of(0.5f * (lo[a] + hi[a]), cl, ch - cl);
            const uint32_t k = seg * 3 * kBins + b;
            // a warp whose primitives all fall into one bin (neighbours in a mesh, near the
            // root) reduces in registers; otherwise what does not widen the bin is dropped
            const uint32_t k0 = __shfl_sync(any, k, __ffs(any) - 1);
            const int one = __all_sync(any, merged && k == k0);
            if (one) {
                uint32_t v[6];
                for (int c = 0; c < 3; ++c) {
                    v[c] = __reduce_min_sync(any, ol[c]);
                    v[3 + c] = __reduce_max_sync(any, oh[c]);
                }
                if ((threadIdx.x & 31u) == __ffs(any) - 1) {
                    atomicAdd(&sCnt[k], __popc(any));
                    for (int c = 0; c < 3; ++c) {
                        atomicMin(&sLo[k][c], v[c]);
                        atomicMax(&sHi[k][c], v[3 + c]);
                    }
                }
            } else if (merged) {
                atomicAdd(&sCnt[k], 1u);
                for (int c = 0; c < 3; ++c) {
                    if (ol[c] < sLo[k][c]) atomicMin(&sLo[k][c], ol[c]);
                    if (oh[c] > sHi[k][c]) atomicMax(&sHi[k][c], oh[c]);
                }
            } else {
                Bin* bn = bins + (size_t)t * 3 * kBins + b;
                atomicAdd(&bn->cnt, 1u);
                for (int c = 0; c < 3; ++c) {
                    atomicMin(&bn->lo[c], ol[c]);
                    atomicMax(&bn->hi[c], oh[c]);
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < numSeg * 3 * kBins; k += blockDim.x) {
        if (!sCnt[k]) continue;
        Bin* bn = bins + (size_t)segTask[k / (3 * kBins)] * 3 * kBins + k % (3 * kBins);
        atomicAdd(&bn->cnt, sCnt[k]);
        for (int c = 0; c < 3; ++c) {
            atomicMin(&bn->lo[c], sLo[k][c]);
            atomicMax(&bn->hi[c], sHi[k][c]);
        }
    }
}

__device__ __forceinline__ float half_area(const float lo[3], const float hi[3]) {
    float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
    if (!(dx >= 0.0f)) return 0.0f;
    return dx * dy + dy * dz + dz * dx;
}

// One warp per task: a half-warp holds the 16 bins of an axis, and the areas and counts on
// both sides of every plane come from its prefix and suffix scans (one thread per task
// walked 48 bins one after the other: 945 us of a 676k-triangle build, now 267).
// The lowest cost wins, the lower axis and plane on ties.
__global__ void __launch_bounds__(128) k_split(const Task* __restrict__ tasks, Bin* __restrict__ bins, Split* splits,
                                               Task* nextTasks, OBox* nextCen, SmallTask* small, BNode* nodes, OBox* nbox,
                                               uint8_t* fromLevels, BuildCtr* ctr) {
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (t >= ctr->cur) return;  // (warp-uniform)
    const uint32_t full = 0xffffffffu, bin = lane & 15u;
    float bestCost = FLT_MAX;
    uint32_t bestKey = 0xffffffffu, bestLeft = 0;
#pragma unroll
    for (uint32_t pass = 0; pass < 2; ++pass) {  // axes 0 and 1, then axis 2 (in both halves)
        const uint32_t axis = pass ? 2u : lane >> 4;
        Bin* B = bins + ((size_t)t * 3 + axis) * kBins + bin;
        const uint4 w0 = reinterpret_cast<const uint4*>(B)[0], w1 = reinterpret_cast<const uint4*>(B)[1];
        float pl[3] = {o2f(w0.y), o2f(w0.z), o2f(w0.w)}, ph[3] = {o2f(w1.x), o2f(w1.y), o2f(w1.z)};
        float sl[3] = {pl[0], pl[1], pl[2]}, sh[3] = {ph[0], ph[1], ph[2]};
        uint32_t pc = w0.x, sc = w0.x;
        __syncwarp();
        clear_bin(B);
#pragma unroll
        for (uint32_t o = 1; o < 16; o <<= 1) {
            const uint32_t c0 = __shfl_up_sync(full, pc, o, 16), c1 = __shfl_down_sync(full, sc, o, 16);
            const bool up = bin >= o, down = bin + o < 16;
            if (up) pc += c0;
            if (down) sc += c1;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float a0 = __shfl_up_sync(full, pl[k], o, 16), a1 = __shfl_up_sync(full, ph[k], o, 16);
                const float b0 = __shfl_down_sync(full, sl[k], o, 16), b1 = __shfl_down_sync(full, sh[k], o, 16);
                if (up) { pl[k] = fminf(pl[k], a0); ph[k] = fmaxf(ph[k], a1); }
                if (down) { sl[k] = fminf(sl[k], b0); sh[k] = fmaxf(sh[k], b1); }
            }
        }
        // the plane behind this bin: the suffix of the next one lies right of it
        const float rightA = __shfl_down_sync(full, half_area(sl, sh), 1, 16);
        const uint32_t rightN = __shfl_down_sync(full, sc, 1, 16);
        if (bin < kBins - 1 && pc != 0 && rightN != 0) {
            const float cost = half_area(pl, ph) * (float)pc + rightA * (float)rightN;
            if (cost < bestCost) {
                bestCost = cost;
                bestKey = axis * kBins + bin;
                bestLeft = pc;
            }
        }
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1) {
        const float c = __shfl_xor_sync(full, bestCost, o);
        const uint32_t k = __shfl_xor_sync(full, bestKey, o), l = __shfl_xor_sync(full, bestLeft, o);
        if (c < bestCost || (c == bestCost && k < bestKey)) {
            bestCost = c;
            bestKey = k;
            bestLeft = l;
        }
    }
    if (lane != 0) return;
    const int bestAxis = bestKey == 0xffffffffu ? -1 : (int)(bestKey / kBins), bestBin = (int)(bestKey % kBins);
    const Task tk = tasks[t];
    const uint32_t cnt = tk.end - tk.begin;
    Split sp;
    sp.axis = bestAxis;
    sp.bin = bestBin;
    sp.nLeft = bestAxis >= 0 ? bestLeft : cnt / 2;  // object median when no plane separates
    uint32_t child = atomicAdd(&ctr->nodes, 2u);
    sp.leftNode = child;
    BNode nd;
    nd.left = child;
    nd.count = 0;
    nodes[tk.node] = nd;  // box filled from nbox at the end
    fromLevels[tk.node] = 1;
    fromLevels[child] = 1;
    fromLevels[child + 1] = 1;
    uint32_t nn[2] = {sp.nLeft, cnt - sp.nLeft};
    uint32_t beg[2] = {tk.begin, tk.begin + sp.nLeft};
    int tid[2];
    for (int s = 0; s < 2; ++s) {
        OBox e;
        obox_empty(e);
        nbox[child + s] = e;
        if (nn[s] > kSmallTask) {
            uint32_t q = atomicAdd(&ctr->nextTasks, 1u);
            Task nt;
            nt.node = child + s;
            nt.begin = beg[s];
            nt.end = beg[s] + nn[s];
            nt.pad = 0;
            nextTasks[q] = nt;
            nextCen[q] = e;
            tid[s] = (int)q;
        } else {
            uint32_t q = atomicAdd(&ctr->small, 1u);
            SmallTask st;
            st.node = child + s;
            st.begin = beg[s];
            st.end = beg[s] + nn[s];
            st.pad = 0;
            small[q] = st;
            tid[s] = -1;
        }
    }
    sp.leftTask = tid[0];
    sp.rightTask = tid[1];
    splits[t] = sp;
}

__device__ __forceinline__ bool goes_left(const Split& sp, const Task& tk, uint32_t i, const OBox& cb, float4 l,
                                          float4 h) {
    if (sp.axis < 0) return (i - tk.begin) < sp.nLeft;
    float lo = sp.axis == 0 ? l.x : (sp.axis == 1 ? l.y : l.z);
    float hi = sp.axis == 0 ? h.x : (sp.axis == 1 ? h.y : h.z);
    float cl = o2f(cb.lo[sp.axis]), ch = o2f(cb.hi[sp.axis]);
    return bin_of(0.5f * (lo + hi), cl, ch - cl) <= sp.bin;
}

__global__ void k_flags(uint32_t n, const uint32_t* __restrict__ ref, const int* __restrict__ taskOf,
                        const Task* __restrict__ tasks, const OBox* __restrict__ tcen, const Split* __restrict__ splits,
                        const float4* __restrict__ blo, const float4* __restrict__ bhi, uint32_t* flags) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int t = taskOf[i];
    uint32_t f = 0;
    if (t >= 0) {
        uint32_t p = ref[i];
        f = goes_left(splits[t], tasks[t], i, tcen[t], blo[p], bhi[p]) ? 1u : 0u;
    }
    flags[i] = f;
}

__global__ void __launch_bounds__(256) k_scatter(uint32_t n, const uint32_t* __restrict__ ref, const int* __restrict__ taskOf,
                          const Task* __restrict__ tasks, const OBox* __restrict__ tcen,
                          const Split* __restrict__ splits, const float4* __restrict__ blo,
                          const float4* __restrict__ bhi, const uint32_t* __restrict__ flags,
                          const uint32_t* __restrict__ scan, uint32_t* ref2, int* taskOf2, OBox* nextCen, OBox* nbox) {
    // per segment [side][lo xyz | hi xyz] of the two children's boxes, then of their centroid
    // bounds (block_segment)
    __shared__ uint32_t sBox[kBoxSegments][24];
    __shared__ int segTask[kBoxSegments];
    uint32_t numSeg;
    const uint32_t seg = block_segment(n, taskOf, kBoxSegments, segTask, &numSeg);
    for (uint32_t k = threadIdx.x; k < numSeg * 24; k += blockDim.x) sBox[k / 24][k % 24] = (k % 6) < 3 ? 0xffffffffu : 0u;
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const int t = taskOf[i];
        const uint32_t p = ref[i];
        if (t < 0) {
            ref2[i] = p;
            taskOf2[i] = -1;
        } else {
            const Task tk = tasks[t];
            const Split sp = splits[t];
            const uint32_t base = scan[tk.begin];
            const uint32_t lr = scan[i] - base;
            const bool left = flags[i] != 0;
            const uint32_t np = left ? tk.begin + lr : tk.begin + sp.nLeft + ((i - tk.begin) - lr);
            ref2[np] = p;
            const int nt = left ? sp.leftTask : sp.rightTask;
            taskOf2[np] = nt;
            const uint32_t node = sp.leftNode + (left ? 0 : 1), side = left ? 0u : 1u;
            const float4 l = blo[p], h = bhi[p];
            const float lo[3] = {l.x, l.y, l.z}, hi[3] = {h.x, h.y, h.z};
            const bool merged = seg < kBoxSegments;
            uint32_t* bx = merged ? &sBox[seg][side * 6] : nullptr;
            uint32_t* cx = merged ? &sBox[seg][12 + side * 6] : nullptr;
            for (int k = 0; k < 3; ++k) {
                const uint32_t l = f2o(lo[k]), h = f2o(hi[k]), c = f2o(0.5f * (lo[k] + hi[k]));
                if (!merged) {
                    atomicMin(&nbox[node].lo[k], l);
                    atomicMax(&nbox[node].hi[k], h);
                    if (nt >= 0) {
                        atomicMin(&nextCen[nt].lo[k], c);
                        atomicMax(&nextCen[nt].hi[k], c);
                    }
                } else {
                    if (l < bx[k]) atomicMin(&bx[k], l);
                    if (h > bx[3 + k]) atomicMax(&bx[3 + k], h);
                    if (c < cx[k]) atomicMin(&cx[k], c);
                    if (c > cx[3 + k]) atomicMax(&cx[3 + k], c);
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < numSeg * 24; j += blockDim.x) {
        const uint32_t k = j % 24, side = (k / 6) & 1u, f = k % 6;
        const int t = segTask[j / 24];
        const bool lo = f < 3;
        const uint32_t v = sBox[j / 24][k];
        if (t < 0 || v == (lo ? 0xffffffffu : 0u)) continue;  // nothing of this side passed through
        const Split& sp = splits[t];
        OBox* o;
        if (k < 12) {
            o = &nbox[sp.leftNode + side];
        } else {
            const int nt = side ? sp.rightTask : sp.leftTask;
            if (nt < 0) continue;
            o = &nextCen[nt];
        }
        if (lo) atomicMin(&o->lo[f], v);
        else atomicMax(&o->hi[f - 3], v);
    }
}

// A half-warp finishes a small task, one primitive per lane: every open node of the task
// is a segment [sb, se) of the lanes, and each round splits all of them at the lowest SAH
// cost over the three orders sorted by centroid (rank by counting, stable; areas of both
// sides by segmented scans).  One thread per task, with its sort and its stack in local
// memory, waited on dependent loads: 585 us for a 676k-triangle build, now 213.
constexpr int kSmallThreads = 128;
__global__ void __launch_bounds__(kSmallThreads) k_small(uint32_t numSmall, const SmallTask* __restrict__ small, uint32_t* ref,
                                                         const float4* __restrict__ blo, const float4* __restrict__ bhi,
                                                         BNode* nodes, BuildCtr* ctr) {
    static_assert(kSmallTask == 16, "a half-warp holds a small task");
    constexpr uint32_t full = 0xffffffffu;
    __shared__ float sBox[kSmallThreads / 32][6][32];
    __shared__ uint32_t sId[kSmallThreads / 32][32];
    const uint32_t lane = threadIdx.x & 31u, h = lane & 15u, base = lane & 16u, warp = threadIdx.x >> 5;
    const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    if (((blockIdx.x * blockDim.x + threadIdx.x) & ~31u) >> 4 >= numSmall) return;  // (warp-uniform)
    SmallTask st{0, 0, 0, 0};
    if (s < numSmall) st = small[s];
    const uint32_t total = st.end - st.begin;
    // this lane's segment (lanes of the half-warp) and its node; a closed lane is its own
    uint32_t sb = 0, se = total, node = st.node, id = 0;
    bool open = h < total;
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    if (open) {
        id = ref[st.begin + h];
        const float4 l = blo[id], u = bhi[id];
        lo[0] = l.x; lo[1] = l.y; lo[2] = l.z;
        hi[0] = u.x; hi[1] = u.y; hi[2] = u.z;
    } else {
        sb = h;
        se = h + 1;
    }
    while (__any_sync(full, open)) {
        const uint32_t cnt = se - sb;
        float bestCost = FLT_MAX;
        uint32_t bestKey = 0xffffffffu, ranks = 0;  // key: axis, then how many lie left of the plane
        float parentA = 0.0f, nlo[3], nhi[3];
#pragma unroll
        for (uint32_t a = 0; a < 3; ++a) {
            const uint32_t key = f2o(lo[a] + hi[a] + 0.0f);  // (-0 and 0 tie)
            uint32_t rank = sb;
            for (uint32_t k = 0; k < 16; ++k) {
                const uint32_t o = __shfl_sync(full, key, k, 16);
                rank += k >= sb && k < se && (o < key || (o == key && k < h)) ? 1u : 0u;
            }
            ranks |= rank << (8 * a);
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sBox[warp][c][base + rank] = lo[c];
                sBox[warp][3 + c][base + rank] = hi[c];
            }
            __syncwarp();
            float pl[3], ph[3], sl[3], sh[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                pl[c] = sl[c] = sBox[warp][c][lane];
                ph[c] = sh[c] = sBox[warp][3 + c][lane];
            }
#pragma unroll
            for (uint32_t o = 1; o < 16; o <<= 1) {
                const bool up = h >= sb + o, down = h + o < se;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float a0 = __shfl_up_sync(full, pl[c], o, 16), a1 = __shfl_up_sync(full, ph[c], o, 16);
                    const float b0 = __shfl_down_sync(full, sl[c], o, 16), b1 = __shfl_down_sync(full, sh[c], o, 16);
                    if (up) { pl[c] = fminf(pl[c], a0); ph[c] = fmaxf(ph[c], a1); }
                    if (down) { sl[c] = fminf(sl[c], b0); sh[c] = fmaxf(sh[c], b1); }
                }
            }
            if (a == 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    nlo[c] = __shfl_sync(full, pl[c], se - 1, 16);
                    nhi[c] = __shfl_sync(full, ph[c], se - 1, 16);
                }
                parentA = half_area(nlo, nhi);
            }
            const float rightA = __shfl_down_sync(full, half_area(sl, sh), 1, 16);
            const uint32_t left = h - sb + 1;
            if (left < cnt) {
                const float cost = half_area(pl, ph) * (float)left + rightA * (float)(cnt - left);
                if (cost < bestCost) {
                    bestCost = cost;
                    bestKey = a * 16 + left;
                }
            }
        }
#pragma unroll
        for (uint32_t o = 1; o < 16; o <<= 1) {  // the segment's last lane gets its best
            const float c = __shfl_up_sync(full, bestCost, o, 16);
            const uint32_t k = __shfl_up_sync(full, bestKey, o, 16);
            if (h >= sb + o && (c < bestCost || (c == bestCost && k < bestKey))) {
                bestCost = c;
                bestKey = k;
            }
        }
        bestCost = __shfl_sync(full, bestCost, se - 1, 16);
        bestKey = __shfl_sync(full, bestKey, se - 1, 16);
        const bool found = bestKey != 0xffffffffu;
        // into the best order, whether the node is split or becomes a leaf
        const uint32_t to = base + (found ? (ranks >> (8 * (bestKey >> 4))) & 0xffu : h);
        __syncwarp();
        sId[warp][to] = id;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sBox[warp][c][to] = lo[c];
            sBox[warp][3 + c][to] = hi[c];
        }
        __syncwarp();
        id = sId[warp][lane];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = sBox[warp][c][lane];
            hi[c] = sBox[warp][3 + c][lane];
        }
        // leaf when small enough and the split does not pay for a traversal step,
        // priced at half a triangle test (SAH with Ct/Ci = 0.5: an 8-wide node test
        // is shared by up to eight children; showcase extension traversal ran 3.5 % faster
        // than with Ct/Ci = 1)
        bool leaf = cnt <= 1 ||
                    (cnt <= kMaxLeaf && (parentA <= 0.0f || (float)cnt * parentA <= 0.5f * parentA + bestCost));
        if (!found) leaf = cnt <= kMaxLeaf;
        const uint32_t pos = found ? bestKey & 15u : cnt / 2;
        const bool head = open && h == sb;
        const uint32_t split = __ballot_sync(full, head && !leaf);
        uint32_t child = 0;
        if (lane == 0 && split) child = atomicAdd(&ctr->nodes, 2u * __popc(split));
        child = __shfl_sync(full, child, 0) + 2u * __popc(split & ((1u << (base + sb)) - 1u));
        if (head) {
            BNode nd;
            for (int c = 0; c < 3; ++c) { nd.lo[c] = nlo[c]; nd.hi[c] = nhi[c]; }
            nd.left = leaf ? st.begin + sb : child;
            nd.count = leaf ? cnt : 0;
            nodes[node] = nd;
        }
        if (!open) continue;
        if (leaf) {
            open = false;
            sb = h;
            se = h + 1;
        } else if (h < sb + pos) {
            se = sb + pos;
            node = child;
        } else {
            sb += pos;
            node = child + 1;
        }
    }
    if (h < total) ref[st.begin + h] = id;
}

// Boxes of level-built nodes live in nbox (atomics); small-task nodes wrote theirs.
__global__ void k_fix_boxes(uint32_t numNodes, BNode* nodes, const OBox* __restrict__ nbox,
                            const uint8_t* __restrict__ fromLevels) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= numNodes || !fromLevels[i]) return;
    for (int k = 0; k < 3; ++k) {
        nodes[i].lo[k] = o2f(nbox[i].lo[k]);
        nodes[i].hi[k] = o2f(nbox[i].hi[k]);
    }
}

// ---------------------------------------------------------------------------
// Collapse to 8-wide compressed nodes.
struct CItem {
    uint32_t bnode, onode;
};

__device__ __forceinline__ float node_area(const BNode& b) {
    float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    return dx * dy + dy * dz + dz * dx;
}

// One thread, before each collapse depth: last depth's new nodes become this one's items.
__global__ void k_collapse_begin(CollapseCtr* ctr) {
    ctr->cur = ctr->next;
    ctr->next = 0;
}

// Eight lanes per node, a child each: what was a chain of loads, double-precision logarithms
// and 64-entry searches in one thread (40-65 us a depth however few its nodes, 547 us of a
// 676k-triangle build, now 193) runs over the lanes, and a warp's four nodes share their atomics.
// Scaling by a power of two is exact, so the boxes are those of the division by it.
__global__ void __launch_bounds__(128) k_collapse(const CItem* __restrict__ items, const BNode* __restrict__ bn,
                                                  const uint32_t* __restrict__ ref, const float* __restrict__ vtx,
                                                  const uint32_t* __restrict__ idx, const uint32_t* __restrict__ triMat,
                                                  uint4* onodes, float4* otris, CItem* next, CollapseCtr* ctr, uint32_t depth) {
    constexpr uint32_t full = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, c = lane & 7u, base = lane & 24u;
    const uint32_t cur = ctr->cur;
    // (a grid capped at what is resident: its bound is up to 512 times the items of a depth)
    for (uint32_t first = ((blockIdx.x * blockDim.x + threadIdx.x) & ~31u) >> 3; first < cur; first += gridDim.x * blockDim.x >> 3) {
        const uint32_t item = first + (lane >> 3);
        const bool live = item < cur;
        const CItem it = live ? items[item] : CItem{0, 0};
        const BNode root = bn[it.bnode];
        // open the child of the largest area (the first of equals) until there are eight
        uint32_t n = !live ? 0 : root.count > 0 ? 1 : 2, kid = root.count > 0 ? it.bnode : root.left + c;
        BNode kb{};
        if (c < n) kb = bn[kid];
        for (int round = 0; round < 6; ++round) {
            float a = c < n && kb.count == 0 ? node_area(kb) : -1.0f;
            if (!(a > -1.0f)) a = -1.0f;
            uint32_t j = c;
#pragma unroll
            for (uint32_t o = 4; o > 0; o >>= 1) {
                const float a1 = __shfl_xor_sync(full, a, o);
                const uint32_t j1 = __shfl_xor_sync(full, j, o);
                if (a1 > a || (a1 == a && j1 < j)) { a = a1; j = j1; }
            }
            const bool grow = n < 8 && a > -1.0f;  // (the same in the node's lanes)
            if (!__any_sync(full, grow)) break;
            const uint32_t left = __shfl_sync(full, kb.left, j, 8);
            if (grow) {
                if (c == j || c == n) {
                    kid = left + (c == n ? 1 : 0);
                    kb = bn[kid];
                }
                ++n;
            }
        }
        // node box and child centroids
        float lo[3], hi[3], d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = c < n ? kb.lo[k] : FLT_MAX;
            hi[k] = c < n ? kb.hi[k] : -FLT_MAX;
#pragma unroll
            for (uint32_t o = 4; o > 0; o >>= 1) {
                lo[k] = fminf(lo[k], __shfl_xor_sync(full, lo[k], o));
                hi[k] = fmaxf(hi[k], __shfl_xor_sync(full, hi[k], o));
            }
            d[k] = 0.5f * (kb.lo[k] + kb.hi[k]) - 0.5f * (lo[k] + hi[k]);
        }
        // slot s takes the child lying furthest toward corner s (bit k set = negative side of
        // axis k): the best pair of a free slot and an unplaced child, until all are placed
        uint32_t taken = 0, src = 8;  // src: the child of slot c
        bool placed = c >= n;
        for (uint32_t round = 0; __any_sync(full, round < n); ++round) {
            float best = -INFINITY;
            uint32_t key = 64 + c * 8;
            if (!placed) {
                best = -FLT_MAX;
                key = c * 8 + __ffs(~taken) - 1;
#pragma unroll
                for (uint32_t s = 0; s < 8; ++s) {
                    const float cost = ((s & 1) ? -d[0] : d[0]) + ((s & 2) ? -d[1] : d[1]) + ((s & 4) ? -d[2] : d[2]);
                    if (!((taken >> s) & 1u) && cost > best) { best = cost; key = c * 8 + s; }
                }
            }
#pragma unroll
            for (uint32_t o = 4; o > 0; o >>= 1) {
                const float b1 = __shfl_xor_sync(full, best, o);
                const uint32_t k1 = __shfl_xor_sync(full, key, o);
                if (b1 > best || (b1 == best && k1 < key)) { best = b1; key = k1; }
            }
            if (round < n) {
                const uint32_t j = key >> 3, s = key & 7u;
                taken |= 1u << s;
                if (c == j) placed = true;
                if (c == s) src = j;
            }
        }
        // from here on a lane is a slot
        const bool have = src < 8;
        const uint32_t from = have ? src : c;
        BNode b;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            b.lo[k] = __shfl_sync(full, kb.lo[k], from, 8);
            b.hi[k] = __shfl_sync(full, kb.hi[k], from, 8);
        }
        b.left = __shfl_sync(full, kb.left, from, 8);
        b.count = __shfl_sync(full, kb.count, from, 8);
        kid = __shfl_sync(full, kid, from, 8);
        const bool inner = have && b.count == 0;
        const uint32_t inners = __ballot_sync(full, inner), imask = (inners >> base) & 0xffu;
        const uint32_t tris = have && !inner ? b.count : 0;
        uint32_t upto = tris;  // triangles of this warp's slots up to this one
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(full, upto, o);
            if (lane >= o) upto += v;
        }
        uint32_t nodes0 = 0, next0 = 0, tris0 = 0;
        if (lane == 31) {
            if (inners) {
                nodes0 = atomicAdd(&ctr->nodes, __popc(inners));
                next0 = atomicAdd(&ctr->next, __popc(inners));
                atomicMax(&ctr->maxDepth, depth + 1);
            }
            if (upto) tris0 = atomicAdd(&ctr->tris, upto);
        }
        const uint32_t before = __popc(inners & ((1u << base) - 1u)), rank = __popc(imask & ((1u << c) - 1u));
        nodes0 = __shfl_sync(full, nodes0, 31) + before;
        const uint32_t childBase = imask ? nodes0 : 0;
        next0 = __shfl_sync(full, next0, 31) + before;
        tris0 = __shfl_sync(full, tris0, 31);
        const uint32_t groupFirst = __shfl_sync(full, upto - tris, 0, 8), groupLast = __shfl_sync(full, upto, 7, 8);
        const uint32_t triBase = groupLast != groupFirst ? tris0 + groupFirst : 0, triOff = upto - tris - groupFirst;
        // quantization frame: step >= 2^-20 of the coordinate magnitude
        auto exponent = [](double x) { return (int)((__double_as_longlong(x) >> 52) & 0x7ff) - 1023; };
        auto pow2 = [](int e) { return __longlong_as_double((long long)(1023 + e) << 52); };
        uint32_t word[7], eb = imask << 24;  // meta, qlo xyz, qhi xyz: this slot's byte, then its half of the node's
        for (int k = 0; k < 3; ++k) {
            const double ext = (double)hi[k] - (double)lo[k];
            const double mag = fmax(fabs((double)lo[k]), fabs((double)hi[k]));
            int e = -126;
            if (ext > 0.0) {
                const double r = ext / 255.0;
                e = exponent(r) + ((__double_as_longlong(r) & 0xfffffffffffffll) ? 1 : 0);
            }
            if (mag > 0.0 && e < exponent(mag) - 20) e = max(e, (int)floor(log2(mag)) - 20);  // (flat nodes only)
            e = max(-126, min(127, e));
            while (e < 127 && ext * pow2(-e) > 253.0) ++e;  // room for the one-step widening
            const double inv = pow2(-e);
            const double ql = floor(((double)b.lo[k] - (double)lo[k]) * inv) - 1.0;
            const double qh = ceil(((double)b.hi[k] - (double)lo[k]) * inv) + 1.0;
            word[1 + k] = have ? (uint32_t)(uint8_t)fmax(0.0, fmin(255.0, ql)) : 255u;
            word[4 + k] = have ? (uint32_t)(uint8_t)fmax(0.0, fmin(255.0, qh)) : 0u;
            eb |= (uint32_t)(e + 127) << (8 * k);
        }
        word[0] = tris ? triOff | ((tris - 1u) << 5) : 0u;
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            uint32_t v = word[k] << (8 * (c & 3u));
            v |= __shfl_xor_sync(full, v, 1);
            v |= __shfl_xor_sync(full, v, 2);
            word[k] = v;
        }
        if (!live) continue;
        if (inner) next[next0 + rank] = {kid, childBase + rank};
        uint32_t* o = reinterpret_cast<uint32_t*>(onodes + 5 * (size_t)it.onode);
        if ((c & 3u) == 0) {  // lanes 0 and 4 hold the two halves
#pragma unroll
            for (int k = 0; k < 7; ++k) o[6 + 2 * k + (c >> 2)] = word[k];
        }
        if (c == 1) *reinterpret_cast<uint4*>(o) = make_uint4(__float_as_uint(lo[0]), __float_as_uint(lo[1]), __float_as_uint(lo[2]), eb);
        if (c == 2) *reinterpret_cast<uint2*>(o + 4) = make_uint2(childBase, triBase);
        for (uint32_t k = 0; k < tris; ++k) {
            const uint32_t p = ref[b.left + k];
            const uint32_t i0 = idx[3 * p], i1 = idx[3 * p + 1], i2 = idx[3 * p + 2];
            const float ax = vtx[3 * i0], ay = vtx[3 * i0 + 1], az = vtx[3 * i0 + 2];
            const float bx = vtx[3 * i1], by = vtx[3 * i1 + 1], bz = vtx[3 * i1 + 2];
            const float cx = vtx[3 * i2], cy = vtx[3 * i2 + 1], cz = vtx[3 * i2 + 2];
            float4* t = otris + 3 * (size_t)(triBase + triOff + k);
            t[0] = make_float4(ax, ay, az, __uint_as_float(p));
            t[1] = make_float4(__fsub_rn(bx, ax), __fsub_rn(by, ay), __fsub_rn(bz, az), __uint_as_float(triMat[p]));
            t[2] = make_float4(__fsub_rn(cx, ax), __fsub_rn(cy, ay), __fsub_rn(cz, az), 0.0f);
        }
    }
}

inline unsigned grid_for(uint64_t n, unsigned b) { return (unsigned)((n + b - 1) / b); }

// SAH cost of the 8-wide tree: one node test for the root plus, for every child
// box, its surface area over the root's times the work a ray entering it does
// (one node test, or the leaf's triangle tests).  One thread per node decodes the
// node's quantized child boxes; sums[0] += area x work, sums[1] = the root's area
// (the union of its children).
__device__ double node_sah(const uint4* __restrict__ nodes, uint32_t i, double* sums) {
    const uint4* n = nodes + 5 * (size_t)i;
    const uint4 n0 = n[0], n1 = n[1], n2 = n[2], n3 = n[3], n4 = n[4];
    const float p[3] = {__uint_as_float(n0.x), __uint_as_float(n0.y), __uint_as_float(n0.z)};
    float sc[3];
    for (int a = 0; a < 3; ++a) sc[a] = ldexpf(1.0f, (int)((n0.w >> (8 * a)) & 0xffu) - 127);
    const uint32_t imask = n0.w >> 24;
    const uint32_t qlo[3][2] = {{n2.x, n2.y}, {n2.z, n2.w}, {n3.x, n3.y}};
    const uint32_t qhi[3][2] = {{n3.z, n3.w}, {n4.x, n4.y}, {n4.z, n4.w}};
    float ulo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, uhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    double acc = 0.0;
    for (int s = 0; s < 8; ++s) {
        float lo[3], hi[3];
        bool empty = false;
        for (int a = 0; a < 3; ++a) {
            const uint32_t bl = (qlo[a][s >> 2] >> (8 * (s & 3))) & 0xffu, bh = (qhi[a][s >> 2] >> (8 * (s & 3))) & 0xffu;
            if (bl > bh) empty = true;
            lo[a] = p[a] + (float)bl * sc[a];
            hi[a] = p[a] + (float)bh * sc[a];
        }
        if (empty) continue;
        const uint32_t meta = ((s < 4 ? n1.z : n1.w) >> (8 * (s & 3))) & 0xffu;
        const double work = ((imask >> s) & 1u) ? 1.0 : (double)((meta >> 5) + 1u);
        acc += (double)half_area(lo, hi) * work;
        for (int a = 0; a < 3; ++a) { ulo[a] = fminf(ulo[a], lo[a]); uhi[a] = fmaxf(uhi[a], hi[a]); }
    }
    if (i == 0) sums[1] = (double)half_area(ulo, uhi);
    return acc;
}

__global__ void __launch_bounds__(256) k_sah(const uint4* __restrict__ nodes, uint32_t numNodes, double* sums) {
    typedef cub::BlockReduce<double, 256> BR;
    __shared__ typename BR::TempStorage tmp;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const double acc = BR(tmp).Sum(i < numNodes ? node_sah(nodes, i, sums) : 0.0);
    if (threadIdx.x == 0) atomicAdd(&sums[0], acc);
}

}  // namespace

// The build's scratch (primitive references, tasks, bins, the binary tree, ...: a few
// hundred MB for a 2.4M-triangle scene) comes from a stream-ordered memory pool of
// the library's own, one per device, that keeps its memory between builds: no
// cudaMalloc / cudaFree in the build, and a scene built after another reuses the
// same memory.  The finished tree (nodes, triangle records) is allocated with
// cudaMalloc, as it lives with the scene.
cudaError_t scratch_pool(cudaMemPool_t* out) {
    static std::mutex m;
    static cudaMemPool_t pools[64] = {nullptr};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(m);
    if (!pools[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if ((e = cudaMemPoolCreate(&p, &props)) != cudaSuccess) return e;
        unsigned long long keep = ~0ull;  // never hand memory back at synchronisation
        if ((e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) return e;
        pools[dev] = p;
    }
    *out = pools[dev];
    return cudaSuccess;
}

template <class T>
cudaError_t scratch_alloc(T** p, cudaMemPool_t pool, cudaStream_t st, size_t bytes) {
    return cudaMallocFromPoolAsync(reinterpret_cast<void**>(p), bytes, pool, st);
}

#define WRK_BCHECK(x)                                                                               \
    do {                                                                                            \
        cudaError_t e_ = (x);                                                                       \
        if (e_ != cudaSuccess) {                                                                    \
            snprintf(err, errlen, "BVH build: %s at %s:%d", cudaGetErrorString(e_), __FILE__, __LINE__); \
            goto fail;                                                                              \
        }                                                                                           \
    } while (0)

int build_bvh8(const float* d_vtx, const uint32_t* d_idx, const uint32_t* d_triMat, uint32_t n, cudaStream_t st,
               BvhBuildResult* out, char* err, size_t errlen) {
    // scratch
    float4 *blo = nullptr, *bhi = nullptr;
    uint32_t *ref = nullptr, *ref2 = nullptr, *flags = nullptr, *scan = nullptr;
    int *taskOf = nullptr, *taskOf2 = nullptr;
    Task *tasks = nullptr, *ntasks = nullptr;
    OBox *tcen = nullptr, *ncen = nullptr, *nbox = nullptr;
    Bin* bins = nullptr;
    Split* splits = nullptr;
    SmallTask* small = nullptr;
    BNode* nodes = nullptr;
    BuildCtr* ctr = nullptr;
    uint8_t* fromLevels = nullptr;
    void* cubTmp = nullptr;
    size_t cubBytes = 0;
    CItem *items = nullptr, *items2 = nullptr;
    CollapseCtr* cctr = nullptr;
    uint4* onodes = nullptr;
    float4* otris = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    BuildCtr hc{};
    uint32_t numTasks = 1, numBinary = 0, smallCount = 0;
    uint32_t maxTasks = n / (kSmallTask + 1) + 2;
    uint32_t maxNodes = 2 * n + 1;
    int rc = WRK_ERR_CUDA;

    cudaMemPool_t pool = nullptr;
    WRK_BCHECK(scratch_pool(&pool));
    WRK_BCHECK(cudaEventCreate(&e0));
    WRK_BCHECK(cudaEventCreate(&e1));
    WRK_BCHECK(cudaEventRecord(e0, st));
    WRK_BCHECK(scratch_alloc(&blo, pool, st, sizeof(float4) * n));
    WRK_BCHECK(scratch_alloc(&bhi, pool, st, sizeof(float4) * n));
    WRK_BCHECK(scratch_alloc(&ref, pool, st, sizeof(uint32_t) * n));
    WRK_BCHECK(scratch_alloc(&ref2, pool, st, sizeof(uint32_t) * n));
    WRK_BCHECK(scratch_alloc(&flags, pool, st, sizeof(uint32_t) * n));
    WRK_BCHECK(scratch_alloc(&scan, pool, st, sizeof(uint32_t) * std::max<uint32_t>(n, 4u)));  // also the SAH sums (2 doubles)
    WRK_BCHECK(scratch_alloc(&taskOf, pool, st, sizeof(int) * n));
    WRK_BCHECK(scratch_alloc(&taskOf2, pool, st, sizeof(int) * n));
    WRK_BCHECK(scratch_alloc(&tasks, pool, st, sizeof(Task) * maxTasks));
    WRK_BCHECK(scratch_alloc(&ntasks, pool, st, sizeof(Task) * maxTasks));
    WRK_BCHECK(scratch_alloc(&tcen, pool, st, sizeof(OBox) * maxTasks));
    WRK_BCHECK(scratch_alloc(&ncen, pool, st, sizeof(OBox) * maxTasks));
    WRK_BCHECK(scratch_alloc(&bins, pool, st, sizeof(Bin) * 3 * kBins * (size_t)maxTasks));
    WRK_BCHECK(scratch_alloc(&splits, pool, st, sizeof(Split) * maxTasks));
    WRK_BCHECK(scratch_alloc(&small, pool, st, sizeof(SmallTask) * (size_t)(n + 1)));
    WRK_BCHECK(scratch_alloc(&nodes, pool, st, sizeof(BNode) * maxNodes));
    WRK_BCHECK(scratch_alloc(&nbox, pool, st, sizeof(OBox) * maxNodes));
    WRK_BCHECK(scratch_alloc(&fromLevels, pool, st, maxNodes));
    WRK_BCHECK(scratch_alloc(&ctr, pool, st, sizeof(BuildCtr)));
    WRK_BCHECK(cudaMemsetAsync(fromLevels, 0, maxNodes, st));
    WRK_BCHECK(cudaMemsetAsync(ctr, 0, sizeof(BuildCtr), st));
    WRK_BCHECK(cub::DeviceScan::ExclusiveSum(nullptr, cubBytes, flags, scan, (int)n, st));
    WRK_BCHECK(scratch_alloc(&cubTmp, pool, st, cubBytes));

    k_iota<<<std::min(grid_for(n, 256), 148u * 16u), 256, 0, st>>>(ref, n);
    if (n > kSmallTask) k_init_bins<<<std::min(grid_for(3ull * kBins * maxTasks, 256), 148u * 16u), 256, 0, st>>>(bins, 3 * kBins * maxTasks);
    WRK_BCHECK(cudaMemsetAsync(taskOf, 0, sizeof(int) * n, st));
    {
        OBox e;
        for (int k = 0; k < 3; ++k) { e.lo[k] = f2o(FLT_MAX); e.hi[k] = f2o(-FLT_MAX); }
        WRK_BCHECK(cudaMemcpyAsync(nbox, &e, sizeof(OBox), cudaMemcpyHostToDevice, st));
        WRK_BCHECK(cudaMemcpyAsync(tcen, &e, sizeof(OBox), cudaMemcpyHostToDevice, st));
        Task root{0, 0, n, 0};
        WRK_BCHECK(cudaMemcpyAsync(tasks, &root, sizeof(Task), cudaMemcpyHostToDevice, st));
        BuildCtr c0{1, 1, 0, 0};  // the root task is the first level's one task
        WRK_BCHECK(cudaMemcpyAsync(ctr, &c0, sizeof(BuildCtr), cudaMemcpyHostToDevice, st));
    }
    k_prim_bounds<<<grid_for(n, 256), 256, 0, st>>>(d_vtx, d_idx, n, blo, bhi, nbox, tcen);
    WRK_BCHECK(cudaGetLastError());
    if (n <= kSmallTask) {
        SmallTask s0{0, 0, n, 0};
        WRK_BCHECK(cudaMemcpyAsync(small, &s0, sizeof(SmallTask), cudaMemcpyHostToDevice, st));
        BuildCtr c1{1, 0, 1, 0};
        WRK_BCHECK(cudaMemcpyAsync(ctr, &c1, sizeof(BuildCtr), cudaMemcpyHostToDevice, st));
        uint8_t one = 1;
        WRK_BCHECK(cudaMemcpyAsync(fromLevels, &one, 1, cudaMemcpyHostToDevice, st));
        numTasks = 0;
    }
    // Levels run kLevelsPerSync at a time without a host round trip: the device keeps
    // each level's task count (k_level_begin) and the kernels read it there; the host
    // sizes grids for an upper bound (a task opens at most two child tasks) and reads
    // the count back only between batches.  A level with no open task passes every
    // primitive through unchanged, so the batch may overshoot the last level.
    for (uint32_t bound = numTasks, levels = 0; numTasks > 0;) {
        for (int k = 0; k < kLevelsPerSync; ++k, ++levels) {
            k_level_begin<<<1, 1, 0, st>>>(ctr);
            k_bin<<<grid_for(n, 256), 256, 0, st>>>(n, ref, taskOf, tcen, blo, bhi, bins);
            k_split<<<grid_for((uint64_t)bound * 32, 128), 128, 0, st>>>(tasks, bins, splits, ntasks, ncen, small, nodes,
                                                                         nbox, fromLevels, ctr);
            k_flags<<<grid_for(n, 256), 256, 0, st>>>(n, ref, taskOf, tasks, tcen, splits, blo, bhi, flags);
            WRK_BCHECK(cub::DeviceScan::ExclusiveSum(cubTmp, cubBytes, flags, scan, (int)n, st));
            k_scatter<<<grid_for(n, 256), 256, 0, st>>>(n, ref, taskOf, tasks, tcen, splits, blo, bhi, flags, scan,
                                                         ref2, taskOf2, ncen, nbox);
            WRK_BCHECK(cudaGetLastError());
            std::swap(ref, ref2);
            std::swap(taskOf, taskOf2);
            std::swap(tasks, ntasks);
            std::swap(tcen, ncen);
            bound = std::min(maxTasks, 2 * bound);
        }
        WRK_BCHECK(cudaMemcpyAsync(&hc, ctr, sizeof(BuildCtr), cudaMemcpyDeviceToHost, st));
        WRK_BCHECK(cudaStreamSynchronize(st));
        numTasks = hc.nextTasks;
        bound = numTasks;
        if (numTasks > maxTasks || levels > kMaxLevels) {
            snprintf(err, errlen, "BVH build: task overflow or level limit (%u tasks, %u levels)", numTasks, levels);
            rc = WRK_ERR_DEVICE;
            goto fail;
        }
    }
    WRK_BCHECK(cudaMemcpyAsync(&hc, ctr, sizeof(BuildCtr), cudaMemcpyDeviceToHost, st));
    WRK_BCHECK(cudaStreamSynchronize(st));
    smallCount = hc.small;
    k_fix_boxes<<<grid_for(hc.nodes, 256), 256, 0, st>>>(hc.nodes, nodes, nbox, fromLevels);
    if (smallCount) k_small<<<grid_for((uint64_t)smallCount * 16, kSmallThreads), kSmallThreads, 0, st>>>(smallCount, small, ref, blo, bhi, nodes, ctr);
    WRK_BCHECK(cudaGetLastError());
    WRK_BCHECK(cudaMemcpyAsync(&hc, ctr, sizeof(BuildCtr), cudaMemcpyDeviceToHost, st));
    WRK_BCHECK(cudaStreamSynchronize(st));
    numBinary = hc.nodes;

    // ---- collapse ----
    WRK_BCHECK(scratch_alloc(&items, pool, st, sizeof(CItem) * numBinary));
    WRK_BCHECK(scratch_alloc(&items2, pool, st, sizeof(CItem) * numBinary));
    WRK_BCHECK(scratch_alloc(&cctr, pool, st, sizeof(CollapseCtr)));
    // (a wide node is the root or stands for an inner node of the binary tree, which are half of it)
    WRK_BCHECK(cudaMalloc(&onodes, sizeof(uint4) * 5 * ((size_t)numBinary / 2 + 1)));
    WRK_BCHECK(cudaMalloc(&otris, sizeof(float4) * 3 * (size_t)n));
    {
        CItem r{0, 0};
        WRK_BCHECK(cudaMemcpyAsync(items, &r, sizeof(CItem), cudaMemcpyHostToDevice, st));
        CollapseCtr c0{1, 0, 1, 1, 0};  // the root item is the first depth's one item
        WRK_BCHECK(cudaMemcpyAsync(cctr, &c0, sizeof(CollapseCtr), cudaMemcpyHostToDevice, st));
    }
    {
        // as the binary levels: the item count stays on the device, read back every
        // kLevelsPerSync depths; an 8-wide node opens at most 8 items
        uint32_t cnt = 1, depth = 1;
        CollapseCtr hcc{};
        while (cnt > 0) {
            uint32_t bound = cnt;
            for (int k = 0; k < kLevelsPerSync; ++k) {
                k_collapse_begin<<<1, 1, 0, st>>>(cctr);
                k_collapse<<<std::min(grid_for((uint64_t)bound * 8, 128), 148u * 8u), 128, 0, st>>>(items, nodes, ref, d_vtx, d_idx, d_triMat, onodes,
                                                               otris, items2, cctr, depth);
                WRK_BCHECK(cudaGetLastError());
                std::swap(items, items2);
                ++depth;
                bound = std::min(numBinary, 8 * bound);
            }
            WRK_BCHECK(cudaMemcpyAsync(&hcc, cctr, sizeof(CollapseCtr), cudaMemcpyDeviceToHost, st));
            WRK_BCHECK(cudaStreamSynchronize(st));
            cnt = hcc.next;
            if (depth > 256) {
                snprintf(err, errlen, "BVH collapse: depth limit exceeded");
                rc = WRK_ERR_DEVICE;
                goto fail;
            }
        }
        WRK_BCHECK(cudaEventRecord(e1, st));
        // SAH cost of the finished tree (outside the timed build)
        double hs[2] = {0.0, 0.0};
        WRK_BCHECK(cudaMemsetAsync(scan, 0, 2 * sizeof(double), st));
        if (hcc.nodes) k_sah<<<grid_for(hcc.nodes, 256), 256, 0, st>>>(onodes, hcc.nodes, (double*)scan);
        WRK_BCHECK(cudaGetLastError());
        WRK_BCHECK(cudaMemcpyAsync(hs, scan, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
        WRK_BCHECK(cudaStreamSynchronize(st));
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        if (hcc.tris != n) {
            snprintf(err, errlen, "BVH collapse: %u triangles emitted, expected %u", hcc.tris, n);
            rc = WRK_ERR_DEVICE;
            goto fail;
        }
        out->nodes = onodes;
        out->tris = otris;
        out->numNodes = hcc.nodes;
        out->numBinary = numBinary;
        out->depth = hcc.maxDepth;
        out->ms = ms;
        out->sah = hs[1] > 0.0 ? (float)(1.0 + hs[0] / hs[1]) : 0.0f;
        onodes = nullptr;
        otris = nullptr;
        rc = WRK_OK;
    }
fail:
    for (void* p : {(void*)blo, (void*)bhi, (void*)ref, (void*)ref2, (void*)flags, (void*)scan, (void*)taskOf,
                    (void*)taskOf2, (void*)tasks, (void*)ntasks, (void*)tcen, (void*)ncen, (void*)bins, (void*)splits,
                    (void*)small, (void*)nodes, (void*)nbox, (void*)fromLevels, (void*)ctr, cubTmp, (void*)items,
                    (void*)items2, (void*)cctr})
        if (p) cudaFreeAsync(p, st);
    cudaFree(onodes);
    cudaFree(otris);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    return rc;
}

}  // namespace wrk
