// Ray traversal of the 8-wide compressed BVH: closest hit (extension rays) and
// any hit (shadow rays).  Replaces optixTrace with __closesthit__trace /
// __miss__trace (libWR/kernels/trace.cu:17-153,321-323 in trianglestrip/OfflineRenderer);
// there are no RT cores on B200, so traversal is SIMT integer/FP32 work.
//
// The traversal itself is in wrk_trav.cuh.
#include <algorithm>

#include "wrk_trav.cuh"

namespace wrk {

// A warp fetches new rays when fewer lanes than this still have one in flight.  The
// wavefront kernels fetch through one counter, whose cost grows with the number of
// fetches (showcase extension stage 32.8 ms at 16, 33.6 at 18, 38.6 at 24); the query
// kernel's chunks are static, so it refills earlier (1M closest + occlusion queries of a
// 676k-triangle scene 739 us at 16, 703 at 20).
constexpr int kRefillAt = 16, kRefillQuery = 20;
// Resident blocks per SM of the persistent kernels; each grid is that many blocks per SM.
// The kernels wait on L1 / L2 for about a third of their cycles, so blocks pay until the
// registers (65536 / (128 x blocks)) spill: extension traversal of the showcase 32.8 ms
// with 8 blocks (64 registers, no spills), 35.4 with 9 (56, 148 B of spills), 35.4 with
// 7.  A multi-scene lane also carries its scene's pointers.
constexpr int kBlocksExtension = 8, kBlocksShadow = 8, kBlocksMulti = 7, kBlocksQuery = 8;

__device__ __forceinline__ Ray load_ray8(const float* p) {
    float4 a = *reinterpret_cast<const float4*>(p);
    float4 b = *reinterpret_cast<const float4*>(p + 4);
    return Ray{a.x, a.y, a.z, b.x, b.y, b.z, a.w, b.w};
}

// Ray queries: persistent warps, each taking every gridDim-th chunk of 32 rays and
// refilling idle lanes from its chunks (below kRefillQuery busy lanes), so a warp does not
// wait for its slowest ray (one thread per ray ran at 8 of 32 lanes per instruction:
// 1M closest + occlusion queries of a 676k-triangle scene 1022 us, 803 with the refill).
// The chunks are assigned statically.
//
// That suits rays that part ways.  Rays of neighbouring pixels end together, and a warp
// that mixes chunks, or waits behind others in its share of a bright column of the image,
// only loses by it: 2048 x 2048 camera rays of a 676k-triangle scene 885 us with a thread
// per ray scheduled by the hardware, 1248 here (scattered rays: 2178 and 1287).  So a batch of
// several chunks a warp is sampled first, and a coherent one is left to k_query_each, which
// follows.
constexpr uint32_t kQuerySamples = 8;

// Programmatic dependent launch (as the convolutions').
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Eight runs of 32 rays over the batch: are at least six of them bundles, whose origins lie
// within 2 % of the scene's extent (the root's quantization frame) and whose directions
// within an eighth of the first ray's?  (A kernel of its own: in k_query it cost the
// traversal spills, 7 % of scattered batches.)  Clears the query's error word, too.
__global__ void __launch_bounds__(kQuerySamples * 32)
    k_query_sample(const uint4* __restrict__ nodes, const float* __restrict__ rays, uint32_t n, uint32_t* err,
                   uint32_t* sampled) {
    grid_launch_dependents();
    if (threadIdx.x == 0) *err = 0;
    if (!sampled) return;
    const uint32_t lane = threadIdx.x & 31u, sample = threadIdx.x >> 5, e = __ldg(nodes).w;
    const float extent = 256.0f * __uint_as_float(max(max(e & 0xffu, (e >> 8) & 0xffu), (e >> 16) & 0xffu) << 23);
    const uint64_t at = (uint64_t)n * (2 * sample + 1) / (2 * kQuerySamples) & ~31ull;  // (n >= 512)
    const Ray r = load_ray8(rays + 8 * (at + lane));
    auto away = [](float v, float& of) {
        const float first = __shfl_sync(0xffffffffu, v, 0);
        of += fabsf(first);
        return fabsf(v - first);
    };
    float d0 = 0.0f, o0 = 0.0f;
    const float dd = away(r.dx, d0) + away(r.dy, d0) + away(r.dz, d0);
    const float od = away(r.ox, o0) + away(r.oy, o0) + away(r.oz, o0);
    const bool bundle = __all_sync(0xffffffffu, dd <= 0.125f * d0 && od <= 0.02f * extent);
    const uint32_t bundles = __syncthreads_count(lane == 0 && bundle);
    if (threadIdx.x == 0) *sampled = bundles >= kQuerySamples * 3 / 4 ? 1u : 0u;
}

template <bool kAnyHit>
__device__ __forceinline__ void write_answer(const DevScene& s, const Trav& t, uint64_t idx, float* tOut, uint32_t* pOut) {
    const bool hit = t.lBest != kNoHit;
    if (kAnyHit) {
        pOut[idx] = hit ? 1u : 0u;
    } else {
        tOut[idx] = hit ? t.tBest : __int_as_float(0x7f800000);
        pOut[idx] = record_prim(s.tris, t.lBest);
    }
}

template <bool kAnyHit>
__global__ void __launch_bounds__(kTraceBlock, kBlocksQuery)
    k_query(DevScene s, const float* __restrict__ rays, uint32_t n, float* tOut, uint32_t* pOut, uint32_t* err,
            const uint32_t* sampled) {
    grid_wait();
    grid_launch_dependents();
    if (sampled && __ldcg(sampled)) return;
    __shared__ uint2 sstack[kStackSmem * kTraceBlock];
    __shared__ float4 sdir[kTraceBlock];  // the lanes' ray directions | tmin (read by triangle tests only)
    uint2 lstack[kStackLocal];
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t stride = (uint64_t)gridDim.x * kTraceBlock;
    uint64_t next = (uint64_t)blockIdx.x * kTraceBlock + (threadIdx.x & ~31u);
    uint32_t used = 0;  // rays of the chunk at `next` already taken
    const TraceGeom geo{s.nodes, s.tris, s.pairs, s.numNodes, s.numTris};
    Trav t;
    uint32_t idx = 0;
    bool active = false;
    while (true) {
        uint32_t idle;
        while (next < n && (idle = __ballot_sync(0xffffffffu, !active)) != 0) {
            const uint32_t avail = (uint32_t)min((unsigned long long)32u, (unsigned long long)(n - next)) - used;
            const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
            if (!active && rank < avail) {
                idx = (uint32_t)next + used + rank;
                trav_init(t, sdir, load_ray8(rays + 8 * (size_t)idx));
                active = true;
            }
            used += min(avail, (uint32_t)__popc(idle));
            if (used >= 32u || next + used >= n) {
                next += stride;
                used = 0;
            }
        }
        if (!__any_sync(0xffffffffu, active)) break;
        const int refillAt = next < n ? kRefillQuery : 1;
        bool fin = false;
        do {
            if (active && !fin) fin = trav_step<kAnyHit, false>(geo, t, sdir, sstack, lstack, err);
        } while (__popc(__ballot_sync(0xffffffffu, active && !fin)) >= refillAt);
        if (active && fin) {
            write_answer<kAnyHit>(s, t, idx, tOut, pOut);
            active = false;
        }
    }
}

// A thread per ray, for coherent batches.
template <bool kAnyHit>
__global__ void __launch_bounds__(kTraceBlock)
    k_query_each(DevScene s, const float* __restrict__ rays, uint32_t n, float* tOut, uint32_t* pOut, uint32_t* err,
                 const uint32_t* sampled) {
    // launched while k_query drains, which hides the blocks that have nothing to do; one of
    // them ends only after it, and so does this launch
    if (blockIdx.x == 0) grid_wait();
    if (!__ldcg(sampled)) return;  // (written before k_query began, which is all that is known here: read from L2)
    __shared__ uint2 sstack[kStackSmem * kTraceBlock];
    __shared__ float4 sdir[kTraceBlock];
    uint2 lstack[kStackLocal];
    const uint64_t idx = (uint64_t)blockIdx.x * kTraceBlock + threadIdx.x;
    if (idx >= n) return;
    const TraceGeom geo{s.nodes, s.tris, s.pairs, s.numNodes, s.numTris};
    Trav t;
    trav_init(t, sdir, load_ray8(rays + 8 * idx));
    while (!trav_step<kAnyHit, false>(geo, t, sdir, sstack, lstack, err)) {
    }
    write_answer<kAnyHit>(s, t, idx, tOut, pOut);
}

template <bool kAnyHit>
static void launch_query(const DevScene& s, const float* rays, uint32_t n, float* t, uint32_t* out, uint32_t* err,
                         uint32_t* sampled, cudaStream_t st) {
    if (!n) return;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t blocks = (n - 1) / kTraceBlock + 1, resident = (uint32_t)sms * kBlocksQuery;
    // (one chunk a warp needs no choice, which takes 2 us; with two, 262,144 camera rays of a
    // 676k-triangle scene in 8 x 4 tiles take 183 us in k_query and 152 chosen, of 36 triangles 37 and 37)
    const bool choose = blocks > resident;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(std::min(blocks, resident));
    lc.blockDim = dim3(kTraceBlock);
    lc.stream = st;
    lc.attrs = &at;
    lc.numAttrs = 1;
    const uint32_t* flag = choose ? sampled : nullptr;
    k_query_sample<<<1, kQuerySamples * 32, 0, st>>>(s.nodes, rays, n, err, choose ? sampled : nullptr);
    cudaLaunchKernelEx(&lc, k_query<kAnyHit>, s, rays, n, t, out, err, flag);
    lc.gridDim = dim3(blocks);
    if (choose) cudaLaunchKernelEx(&lc, k_query_each<kAnyHit>, s, rays, n, t, out, err, flag);
}

void launch_closest_query(const DevScene& s, const float* rays, uint32_t n, float* t, uint32_t* prim, uint32_t* err,
                          uint32_t* sampled, cudaStream_t st) {
    launch_query<false>(s, rays, n, t, prim, err, sampled, st);
}
void launch_occluded_query(const DevScene& s, const float* rays, uint32_t n, uint32_t* occ, uint32_t* err,
                           uint32_t* sampled, cudaStream_t st) {
    launch_query<true>(s, rays, n, nullptr, occ, err, sampled, st);
}

// ---------------------------------------------------------------------------
// Wavefront trace kernels.  A path's state travels with it: a lane reads its ray
// from the input queue entry it fetched and, when the ray is done, copies the
// whole entry into the next queue at the position a warp-aggregated append (one
// ballot per destination, one atomicAdd by the lowest lane) handed out, so the
// lanes of a warp write consecutive entries.  Queue entries are read and written
// once per pass, so they go through the cache with the streaming (evict-first)
// policy (__ldcs / __stcs) and leave L1 to the BVH nodes and triangle records.
__device__ __forceinline__ PathQ pick_bucket(const Queues& q, uint32_t b) {
    switch (b) {
        case kBucketLambert: return q.bucket[kBucketLambert];
        case kBucketDielectric: return q.bucket[kBucketDielectric];
        case kBucketGGX: return q.bucket[kBucketGGX];
        default: return q.bucket[kBucketOther];
    }
}

// Persistent traversal: each warp keeps its lanes busy by fetching new rays from
// the queue (one warp-aggregated atomic on a per-launch fetch counter) whenever
// fewer than kRefillAt lanes still have a ray in flight, instead of waiting for
// the slowest ray of a fixed batch (Aila & Laine 2009, "Understanding the
// efficiency of ray traversal on GPUs").
template <bool kAnyHit, bool kMulti>
struct TraceBlocks {
    static constexpr int value = kMulti ? kBlocksMulti : (kAnyHit ? kBlocksShadow : kBlocksExtension);
};

__device__ __forceinline__ void count_ended_t(SlotCtl* ctl, bool ended, uint32_t slot) {
    const uint32_t m = __ballot_sync(0xffffffffu, ended);
    if (!m) return;
    const uint32_t peers = __match_any_sync(0xffffffffu, ended ? slot : 0xffffffffu) & m;
    if (ended && (uint32_t)(__ffs(peers) - 1) == (threadIdx.x & 31u))
        atomicAdd(&ctl[slot].finished, (unsigned long long)__popc(peers));
}

// kMulti: the batch's requests may use different scenes; a lane loads the
// geometry of its ray's scene when it fetches the ray.  Otherwise scene s0.
template <bool kAnyHit, bool kMulti>
__global__ void __launch_bounds__(kTraceBlock, (TraceBlocks<kAnyHit, kMulti>::value))
    k_trace_persistent(DevScene s0, Queues q) {
    __shared__ uint2 sstack[kStackSmem * kTraceBlock];
    __shared__ float4 sdir[kTraceBlock];  // the lanes' ray directions | tmin (read by triangle tests only)
    uint2 lstack[kStackLocal];
    Counters* c = q.ctr;
    const uint32_t cur = c->cur;
    const uint32_t n = min(kAnyHit ? c->shd[cur].v : c->ext[cur].v, q.capacity);
    const PathQ in = kAnyHit ? q.shd[cur] : q.ext[cur];
    uint32_t* fetch = kAnyHit ? &c->fetchShadow.v : &c->fetchExtension.v;
    const uint32_t lane = threadIdx.x & 31u;
    // the shadow stage continues every Lambert path it traces (statistics slot)
    if (kAnyHit && blockIdx.x == 0 && threadIdx.x == 0) c->bucket[kBucketLambertResume].v = n;
    // A warp's first rays are the ones at its position in the grid: a queue of at most 32
    // rays per warp never touches the fetch counter (which every warp of the grid, idle
    // ones too, would otherwise visit), and a small one is spread over one warp per
    // scheduler, so that a ray waits for few others.  Later rays come from the counter, as
    // many as there are idle lanes: larger grains per warp measured slower.
    const uint32_t warps = gridDim.x * (kTraceBlock / 32), spread = warps / (TraceBlocks<kAnyHit, kMulti>::value);
    const uint32_t perWarp = min(32u, (n + spread - 1) / spread);
    const uint32_t gridRays = warps * perWarp;
    uint32_t base = (blockIdx.x * (kTraceBlock / 32) + (threadIdx.x >> 5)) * perWarp;
    bool exhausted = base >= n;
    Trav t;
    TraceGeom geo{s0.nodes, s0.tris, s0.pairs, s0.numNodes, s0.numTris};
    uint32_t idx = 0;
    bool active = false;
    while (true) {
        const uint32_t idle = exhausted ? 0u : __ballot_sync(0xffffffffu, !active);
        if (idle) {
            if (base == kInvalidSlot) {
                if (lane == 0) base = atomicAdd(fetch, (uint32_t)__popc(idle)) + gridRays;
                base = __shfl_sync(0xffffffffu, base, 0);
            }
            const bool first = base < gridRays;  // (every lane is idle then)
            idx = active ? idx : base + __popc(idle & ((1u << lane) - 1u));
            if (!active && idx < n && (!first || lane < perWarp)) {
                float4 o = kAnyHit ? __ldcs(in.sh_o + idx) : __ldcs(in.ray_o + idx);
                float4 d = kAnyHit ? __ldcs(in.sh_d + idx) : __ldcs(in.ray_d + idx);
                if constexpr (kMulti) {
                    // a shadow entry keeps its request slot where tmin would be
                    const uint32_t slot = kAnyHit ? __float_as_uint(o.w) : slot_of(__ldcs(&in.st[idx].w));
                    const DevScene& sc = q.scenes[q.req[slot].scene];
                    geo = TraceGeom{sc.nodes, sc.tris, sc.pairs, sc.numNodes, sc.numTris};
                }
                if (kAnyHit) o.w = kShadowTmin;
                trav_init(t, sdir, Ray{o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w});
                active = true;
            }
            exhausted = n <= gridRays || base + __popc(idle) >= n;
            base = kInvalidSlot;
        }
        if (!__any_sync(0xffffffffu, active)) break;
        // once the queue is drained nothing can refill a lane: run to completion
        const int refillAt = exhausted ? 1 : kRefillAt;
        bool fin = false;
        do {
            if (active && !fin) fin = trav_step<kAnyHit, true>(geo, t, sdir, sstack, lstack, &c->error);
        } while (__popc(__ballot_sync(0xffffffffu, active && !fin)) >= refillAt);
        const bool done = active && fin;
        if (kAnyHit) {
            // Shadow stage of __raygen__trace (trace.cu:27-51): add the NEE
            // contribution if nothing lies in [tmin, tmax], then carry out what the
            // Lambert shade decided for the path after its shadow ray: continue
            // with the prepared extension ray, accumulate, or drop.
            uint32_t cont = kContDrop, slot = 0;
            if (done) {
                const float4 cc = __ldcs(in.sh_c + idx);
                const uint32_t w = __float_as_uint(cc.w);
                const bool lit = t.lBest == kNoHit;
                cont = w & 3u;
                slot = __float_as_uint(in.sh_o[idx].w);
                if (cont == kContExt) {
                    // the continuing path's entry waits in the next extension queue
                    const uint32_t pos = w >> 2;
                    if (lit && pos < q.capacity) {
                        const PathQ o = cur ? q.ext[0] : q.ext[1];
                        const float4 rd = o.rad[pos];
                        o.rad[pos] = make_float4(rd.x + cc.x, rd.y + cc.y, rd.z + cc.z, rd.w);
                    }
                } else if (cont == kContAccumulate) {
                    float4 rd = in.rad[idx];
                    if (lit) rd = make_float4(rd.x + cc.x, rd.y + cc.y, rd.z + cc.z, rd.w);
                    const Frame& f = q.req[slot];
                    const float3 L = clamp_fireflies(make_float3(rd.x, rd.y, rd.z), f.fireflyClamp);
                    atomicAdd(f.accum + __float_as_uint(rd.w), make_float4(L.x, L.y, L.z, 0.0f));
                }
            }
            count_ended_t(q.ctl, done && cont != kContExt, slot);
        } else {
            uint32_t bucket = kNumBuckets;
            float4 th = make_float4(0, 0, 0, 0), rd = make_float4(0, 0, 0, 0);
            uint4 st = make_uint4(0, 0, 0, 0);
            bool missed = false;
            uint32_t pBest = kNoHit, mBest = 0;
            if (done) {
                th = __ldcs(in.thr + idx);
                rd = __ldcs(in.rad + idx);
                st = __ldcs(in.st + idx);
                // prim, material and material bucket from the hit's record (just
                // tested, so cached)
                pBest = record_prim(geo.tris, t.lBest);
                mBest = record_material(geo.tris, t.lBest);
                const Frame& f = q.req[slot_of(st.w)];
                const float4 dt = sdir[threadIdx.x];
                const float3 dir = make_float3(dt.x, dt.y, dt.z);
                if (pBest != kNoHit) bucket = __float_as_uint(__ldg(geo.tris + 3 * (size_t)t.lBest + 2).w);
                else if constexpr (kMulti) miss_accumulate(q.scenes[f.scene], f, th, rd, dir);
                else miss_accumulate(s0, f, th, rd, dir);
                missed = pBest == kNoHit;
            }
            count_ended_t(q.ctl, missed, slot_of(st.w));
            // textured Lambert hits fill the Lambert queue from its last entry down
            const bool texL = bucket == (kBucketLambert | kRecTextured);
            if (bucket != kNumBuckets) bucket = texL ? (uint32_t)kBucketLambert : min(bucket, (uint32_t)kBucketOther);
            uint32_t pos = kInvalidSlot;
            // the five appends' atomics are issued together, one by each of lanes 0-4
            const uint32_t dest = texL ? 4u : bucket;
            const uint32_t m0 = __ballot_sync(0xffffffffu, dest == 0u), m1 = __ballot_sync(0xffffffffu, dest == 1u),
                           m2 = __ballot_sync(0xffffffffu, dest == 2u), m3 = __ballot_sync(0xffffffffu, dest == 3u),
                           m4 = __ballot_sync(0xffffffffu, dest == 4u && texL);
            const uint32_t mine = lane == 0 ? m0 : lane == 1 ? m1 : lane == 2 ? m2 : lane == 3 ? m3 : lane == 4 ? m4 : 0u;
            uint32_t base = 0;
            if (mine) base = atomicAdd(lane == 4 ? &c->lambertTex.v : &c->bucket[lane].v, (uint32_t)__popc(mine));
            base = __shfl_sync(0xffffffffu, base, dest & 7u);
            if (bucket != kNumBuckets) {
                const uint32_t peers = dest == 0u ? m0 : dest == 1u ? m1 : dest == 2u ? m2 : dest == 3u ? m3 : m4;
                pos = base + __popc(peers & ((1u << lane) - 1u));
                if (pos >= q.capacity) {
                    atomicOr(&c->error, kErrQueueOverflow);
                    pos = kInvalidSlot;
                } else if (texL) {
                    pos = q.capacity - 1u - pos;
                }
            }
            if (pos != kInvalidSlot) {
                const PathQ o = pick_bucket(q, bucket);
                const float4 dt = sdir[threadIdx.x];
                __stcs(o.ray_o + pos, make_float4(t.ox, t.oy, t.oz, dt.w));
                __stcs(o.ray_d + pos, make_float4(dt.x, dt.y, dt.z, t.tBest));
                o.hit[pos] = make_float4(t.tBest, __uint_as_float(pBest), __uint_as_float(mBest),
                                         __uint_as_float(t.lBest));
                __stcs(o.thr + pos, th);
                __stcs(o.rad + pos, rd);
                __stcs(o.st + pos, st);
            }
        }
        if (done) active = false;
    }
}

void launch_trace_extension(const DevScene& s, const Queues& q, bool multi, int numSMs, cudaStream_t st) {
    if (multi) k_trace_persistent<false, true><<<numSMs * TraceBlocks<false, true>::value, kTraceBlock, 0, st>>>(s, q);
    else k_trace_persistent<false, false><<<numSMs * TraceBlocks<false, false>::value, kTraceBlock, 0, st>>>(s, q);
}
void launch_trace_shadow(const DevScene& s, const Queues& q, bool multi, int numSMs, cudaStream_t st) {
    if (multi) k_trace_persistent<true, true><<<numSMs * TraceBlocks<true, true>::value, kTraceBlock, 0, st>>>(s, q);
    else k_trace_persistent<true, false><<<numSMs * TraceBlocks<true, false>::value, kTraceBlock, 0, st>>>(s, q);
}

}  // namespace wrk
