// BF16 3x3 convolutions on the 5th-generation tensor cores (tcgen05 + TMEM + TMA),
// the compute of the learned denoiser that stands in for libWR's closed OptiX AI
// denoiser (libWR/src/internal/denoiser.cpp:17-195, optixDenoiserInvoke at :171).
//
// Layout: activations NHWC bf16, dense channels (C a multiple of 16); weights
// [Cout][3*3][Cin] bf16 (K-major: k = tap*Cin + ci, tap = dy*3 + dx).
//
// k_conv_fwd  -- implicit GEMM, M = 128 output pixels (an 8 x 16 pixel tile), N = output
//                channels (a multiple of 16, <= 256), K = 9 taps x Cin, from one halo of
//                the input per tile.  Used for the forward pass and, with flipped /
//                transposed weights, for the data gradient.  The epilogue also makes the
//                2x2 average pool, the nearest 2x upsample (four stores) or the network's
//                output image, so those take no passes of their own.
// k_conv_wgrad -- weight gradient dW[co][tap][ci] = sum_p G[p][co] X[p+tap][ci]:
//                M = 3 taps x input channels (128 rows; or 128 input channels of one tap),
//                N = output channels, K = pixels;
//                both operands channel-contiguous (MN-major), the taps are descriptors into
//                one halo.  Split over pixel ranges, f32 atomics into dW.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "conv_tc.h"
#include "tc_conv.cuh"

namespace wrk {
namespace conv {

using namespace tc;

constexpr uint32_t kTileP = 128;  // pixels of a tile

__host__ __device__ constexpr uint32_t round_up(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ---------------------------------------------------------------------------
// Forward convolution (also the data gradient, with flipped / transposed weights).
//
// A work item is one 8 x 16 pixel tile (M = 128) and one slice of N output channels.
// Its input is the tile's 10 x 18 pixel halo, one TMA load per channel chunk (64, 32 or
// 16 channels; zero padding from the out-of-bounds fill), stored K-major with one
// 128 / 64 / 32-byte swizzled row per pixel: the 128 pixels shifted by tap (dy, dx) start
// dy*10 + dx rows in, with the tile's 8-pixel rows (the M core-matrix groups) 10 rows
// apart, so all nine taps are descriptors into the same halo and the input crosses
// L2 -> shared memory once instead of nine times.  The halo chunks form a ring that runs
// across work items, so the next item's input loads while this one computes.
//
// Weights: kResident keeps the layer's whole weight tensor in shared memory; otherwise
// (tap, chunk) slices stream through a second ring.  Where all chunks of a wide input do not
// fit beside a ring of them, the item runs chunk by chunk (kByChunk): nine taps of one
// chunk, then its slot is free for the next, so any channel count does.
//
// Warps: epilogue (four or eight), input loads, MMA, weight loads.  The accumulator is
// double-buffered in TMEM (columns [0, N) and [N, 2N)), so the epilogue of one item
// overlaps the next one's MMAs.  K runs tap-major, then by channel, so every output sums in
// the same order whatever the plan; kByChunk alone runs by chunk, then tap-major.
//
// What bounds it, on a 1920 x 1088 frame (device time per layer, before -> now, with the
// pools and upsamples that were passes of their own, 66 + 178 us, now in it): an M128 K16
// MMA takes 50-60 cycles up to 64 output channels, whatever their number (its 4 KB input
// operand), so 96 -> 32 channels at full resolution takes 287 -> 193 us, the MMAs alone
// 184; the other full-resolution layers waited on their epilogue's 16-byte stores at
// 64-byte strides (32 -> 32 124 us, 65 without the stores) and now leave through shared
// memory and TMA stores (75 us); the layers whose weights do not fit waited on L2 ->
// shared memory traffic, nine copies of the input among it (192 -> 64 202 -> 164 us,
// 384 -> 128 125 -> 96 us) and now wait on their weight slices' MMA steps (315 cycles for
// 200 of MMAs at 64 channels).  The whole frame: 1940 -> 1100 us.
constexpr uint32_t kHaloW = 10, kHaloH = 18, kHaloPix = kHaloW * kHaloH, kHTileW = 8, kHTileH = 16;
// Epilogue warps: four per accumulator buffer for resident layers (one group of four
// alternating between the buffers could not keep up with 9-36 MMAs a tile), four in all
// for streaming ones.
__host__ __device__ constexpr uint32_t fwd_epilogue_warps(bool resident) { return resident ? 8 : 4; }
__host__ __device__ constexpr uint32_t fwd_threads(bool resident) { return (fwd_epilogue_warps(resident) + 3) * 32; }
// Bytes of one channel chunk's halo, padded so that every chunk starts on a swizzle
// pattern boundary.
__host__ __device__ constexpr uint32_t halo_block_bytes(uint32_t chunk) {
    return (kHaloPix * chunk * 2 + 1023) / 1024 * 1024;
}

// Rows of the halo that a weight-gradient block with one or all three rows of taps reads,
// and TMEM columns of one row's sums
__host__ __device__ constexpr uint32_t wgrad_halo_rows(uint32_t rows) { return kHTileH + rows - 1; }
__host__ __device__ constexpr uint32_t wgrad_cols(uint32_t cout) { return (cout + 31) / 32 * 32; }

// ---- epilogue ----
// 16-byte unit u of row r in a staging tile of rowBytes-wide rows, swizzled as the TMA
// store expects it (SWIZZLE_128B / 64B / 32B).
__device__ __forceinline__ uint32_t staged_unit(uint32_t r, uint32_t u, uint32_t rowBytes) {
    const uint32_t x = rowBytes == 128 ? (r & 7u) : rowBytes == 64 ? ((r >> 1) & 3u) : ((r >> 2) & 1u);
    return r * rowBytes + ((u ^ x) << 4);
}
__device__ __forceinline__ void st_shared16(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ uint4 ld_shared16(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t bf2(float a, float b) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    return *(const uint32_t*)&t;
}

// 16 accumulator columns from channel c0 on (channels of this launch's output): bias,
// ReLU, ReLU-derivative mask.
__device__ __forceinline__ void finish16(const Epilogue& ep, const float* bias, uint32_t c0, size_t pix, bool inside,
                                         float (&v)[16]) {
    if (ep.bias) {
#pragma unroll
        for (uint32_t j = 0; j < 16; j += 4) {
            const float4 x = *(const float4*)(bias + c0 + j);
            v[j] += x.x;
            v[j + 1] += x.y;
            v[j + 2] += x.z;
            v[j + 3] += x.w;
        }
    }
    if (ep.relu) {
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.0f);
    }
    if (ep.mask && inside) {
        const __nv_bfloat16* m = ep.mask + pix * ep.maskStride + c0;
        const uint4 a = *(const uint4*)m, b = *(const uint4*)(m + 8);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const float2 f = __bfloat1622float2(*(const __nv_bfloat162*)&w[j]);
            if (!(f.x > 0.0f)) v[2 * j] = 0.0f;
            if (!(f.y > 0.0f)) v[2 * j + 1] = 0.0f;
        }
    }
}

// 16 finished channels, from channel c of the staged slice on, into a staged row
// (rowAddr: the row's first byte; x: its swizzle, already times 16)
__device__ __forceinline__ void stage16(uint32_t rowAddr, uint32_t x, uint32_t c, uint32_t f32, const float (&v)[16]) {
    if (f32) {
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            st_shared16(rowAddr + ((c * 4 + 16 * j) ^ x), __float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]),
                        __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3]));
    } else {
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j)
            st_shared16(rowAddr + ((c * 2 + 16 * j) ^ x), bf2(v[8 * j], v[8 * j + 1]), bf2(v[8 * j + 2], v[8 * j + 3]),
                        bf2(v[8 * j + 4], v[8 * j + 5]), bf2(v[8 * j + 6], v[8 * j + 7]));
    }
}

// 32 accumulator columns: bias, bf16, ReLU (on the rounded pair: rounding keeps the sign),
// into a staged row.
__device__ __forceinline__ void stage32(uint32_t rowAddr, uint32_t x, uint32_t c, const float* bias, uint32_t relu,
                                        const uint32_t (&r)[32]) {
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
        const float4 p = *(const float4*)(bias + 8 * u), q = *(const float4*)(bias + 8 * u + 4);
        uint32_t w[4] = {bf2(__uint_as_float(r[8 * u]) + p.x, __uint_as_float(r[8 * u + 1]) + p.y),
                         bf2(__uint_as_float(r[8 * u + 2]) + p.z, __uint_as_float(r[8 * u + 3]) + p.w),
                         bf2(__uint_as_float(r[8 * u + 4]) + q.x, __uint_as_float(r[8 * u + 5]) + q.y),
                         bf2(__uint_as_float(r[8 * u + 6]) + q.z, __uint_as_float(r[8 * u + 7]) + q.w)};
        if (relu) {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) asm("max.bf16x2 %0, %1, %2;" : "=r"(w[j]) : "r"(w[j]), "r"(0u));
        }
        st_shared16(rowAddr + ((c * 2 + 16 * u) ^ x), w[0], w[1], w[2], w[3]);
    }
}

// The first n of 16 finished channels to element `at` of an output that TMA cannot address
// (rows of no multiple of 16 bytes, or an address of none): 16 bytes a store where they are
// aligned.  (A loop over n indexed the registers through local memory: 64 -> 100 channels
// at 1920 x 1080 2508 us, 776 so.)
__device__ __forceinline__ void store16(const Epilogue& ep, size_t at, uint32_t n, const float (&v)[16]) {
    if (ep.outF32) {
        float* o = (float*)ep.out + at;
        if (n == 16 && ((uintptr_t)o & 15u) == 0) {
#pragma unroll
            for (uint32_t j = 0; j < 16; j += 4) *(float4*)(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j)
                if (j < n) o[j] = v[j];
        }
    } else {
        __nv_bfloat16* o = (__nv_bfloat16*)ep.out + at;
        if (n == 16 && ((uintptr_t)o & 3u) == 0) {
#pragma unroll
            for (uint32_t j = 0; j < 16; j += 2) *(uint32_t*)(o + j) = bf2(v[j], v[j + 1]);
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j)
                if (j < n) o[j] = __float2bfloat16_rn(v[j]);
        }
    }
}

// n / d with inv ~ 1 / d: an estimate and its correction (three integer divisions per
// tile were a fifth of the small layers' epilogue).
__device__ __forceinline__ uint32_t quotient(uint32_t n, uint32_t d, float inv) {
    uint32_t q = __float2uint_rz(__uint2float_rz(n) * inv);
    while ((uint64_t)q * d > n) --q;
    while ((uint64_t)(q + 1) * d <= n) ++q;
    return q;
}
// Image, first row and first column of a work item's tile, and its first output channel.
struct TileAt {
    uint32_t b, h0, w0, n0;
};
__device__ __forceinline__ TileAt tile_at(const FwdShape& sh, uint32_t perImg, float invImg, float invX, uint32_t item) {
    const uint32_t tile = sh.nSplit == 1 ? item : item / sh.nSplit;
    TileAt t;
    t.n0 = (item - tile * sh.nSplit) * sh.N;
    t.b = quotient(tile, perImg, invImg);
    const uint32_t rem = tile - t.b * perImg, ty = quotient(rem, sh.tilesX, invX);
    t.h0 = ty * kHTileH;
    t.w0 = (rem - ty * sh.tilesX) * kHTileW;
    return t;
}

// log1p of the clamped radiance: the network's input scale (and its output's base).
__device__ __forceinline__ float log_radiance(float x) { return log1pf(fmaxf(x, 0.0f)); }

// BLOCKS > 0: the channel chunks of a resident layer, so that the MMA issue is straight
// code with constant descriptor offsets (0 = sh.Cin / CHUNK at run time).
template <int CHUNK, bool kResident, int BLOCKS, bool kByChunk = false>
__global__ void __launch_bounds__(fwd_threads(kResident), kResident && BLOCKS != 3 ? 2 : 1)
    k_conv_fwd(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw,
               const __grid_constant__ OutMaps mo, FwdShape sh, Epilogue ep, uint32_t* err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr uint32_t kRow = CHUNK * 2;  // bytes of a pixel's row of one chunk
    constexpr uint32_t kEpiWarps = fwd_epilogue_warps(kResident);
    constexpr uint32_t kBlock = halo_block_bytes(CHUNK);
    const uint32_t G = BLOCKS > 0 ? BLOCKS : sh.Cin / CHUNK;  // channel chunks
    const uint32_t wSlice = sh.N * kRow;  // bytes of one (tap, chunk) weight slice
    const uint32_t RA = sh.stagesA, RB = sh.stagesB;
    const uint32_t steps = 9 * G;
    // layout: halo ring | weights (resident or ring) | staging | bias | barriers
    const uint32_t base = smem_u32(smem);
    const uint32_t wBase = base + RA * kBlock;
    const uint32_t sBase = wBase + round_up((kResident ? steps : RB) * wSlice, 1024);
    uint8_t* tail = smem + (sBase - base) + sh.stagingBytes * (kEpiWarps / 4);
    float* biasS = (float*)tail;
    uint64_t* bars = (uint64_t*)(tail + 1024);
    // bars: fullA[RA] emptyA[RA] fullB[RB] emptyB[RB] accFull[2] accEmpty[2] drain
    uint32_t* tmemSlot = (uint32_t*)(bars + 2 * RA + 2 * RB + 5);
    volatile uint32_t* abortFlag = tmemSlot + 1;
    auto fullA = [&](uint32_t s) { return smem_u32(bars + s); };
    auto emptyA = [&](uint32_t s) { return smem_u32(bars + RA + s); };
    auto fullB = [&](uint32_t s) { return smem_u32(bars + 2 * RA + s); };
    auto emptyB = [&](uint32_t s) { return smem_u32(bars + 2 * RA + RB + s); };
    auto accFull = [&](uint32_t b) { return smem_u32(bars + 2 * RA + 2 * RB + b); };
    auto accEmpty = [&](uint32_t b) { return smem_u32(bars + 2 * RA + 2 * RB + 2 + b); };
    const uint32_t drain = smem_u32(bars + 2 * RA + 2 * RB + 4);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < 2 * RA + 2 * RB; ++s) mbar_init(smem_u32(bars + s), 1);
        for (uint32_t b = 0; b < 2; ++b) {
            mbar_init(accFull(b), 1);
            mbar_init(accEmpty(b), 4);  // one arrival per epilogue warp
        }
        mbar_init(drain, 1);
        *abortFlag = 0;
        fence_mbar_init();
        prefetch_map(&mx);
        prefetch_map(&mw);
    }
    if (ep.bias)
        for (uint32_t c = threadIdx.x; c < 256; c += blockDim.x) biasS[c] = c < ep.nBias ? ep.bias[c] : 0.0f;
    if (warp == 0) {
        __syncwarp();
        tmem_alloc(smem_u32(tmemSlot), sh.tmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmemSlot;
    // The next launch may set itself up from here on; this one touches what earlier
    // launches produce only after they are done (weights and biases are older: they change
    // between passes, in launches that wait).
    grid_launch_dependents();
    if (warp != kEpiWarps + 2) grid_wait();

    const uint32_t perImg = sh.tilesX * sh.tilesY;
    const uint32_t items = sh.B * perImg * sh.nSplit;
    const float invImg = 1.0f / (float)perImg, invX = 1.0f / (float)sh.tilesX;

    if (warp == kEpiWarps) {
        // input: one halo chunk per ring slot (the whole warp runs the loop, one lane issues)
        const bool leader = elect_one();
        uint32_t s = 0, ph = 1, issued = 0;
        bool ok = true;
        for (uint32_t item = blockIdx.x; ok && item < items; item += gridDim.x) {
            const TileAt at = tile_at(sh, perImg, invImg, invX, item);
            for (uint32_t g = 0; g < G; ++g) {
                if (warp_any(*abortFlag) || !warp_wait(emptyA(s), ph)) {
                    ok = false;
                    break;
                }
                if (leader) {
                    mbar_expect_tx(fullA(s), kHaloPix * kRow);
                    tma_load_4d(base + s * kBlock, &mx, fullA(s), (int)(g * CHUNK), (int)at.w0 - 1, (int)at.h0 - 1,
                                (int)at.b);
                }
                ++issued;
                if (++s == RA) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        if (!ok) {  // let the copies in flight land before the block exits (bounded)
            *abortFlag = 1;
            for (uint32_t j = issued > RA ? issued - RA : 0; j < issued; ++j) mbar_wait(fullA(j % RA), (j / RA) & 1u);
        }
    } else if (warp == kEpiWarps + 2) {
        // weights
        const bool leader = elect_one();
        if (kResident) {
            if (leader) {
                mbar_expect_tx(fullB(0), steps * wSlice);
                for (uint32_t k = 0; k < steps; ++k) tma_load_2d(wBase + k * wSlice, &mw, fullB(0), (int)(k * CHUNK), 0);
            }
            __syncwarp();
            if (!warp_wait(fullB(0), 0)) *abortFlag = 1;
        } else {
            if (leader) {
                uint32_t s = 0, ph = 1, issued = 0;
                bool ok = true;
                for (uint32_t item = blockIdx.x; ok && item < items; item += gridDim.x) {
                    const int row = (int)((item % sh.nSplit) * sh.N);
                    for (uint32_t j = 0; j < steps; ++j) {
                        if (!mbar_wait(emptyB(s), ph)) {
                            ok = false;
                            break;
                        }
                        mbar_expect_tx(fullB(s), wSlice);
                        const uint32_t k = kByChunk ? j % 9 * G + j / 9 : j;  // tap * G + chunk
                        tma_load_2d(wBase + s * wSlice, &mw, fullB(s), (int)(k * CHUNK), row);
                        ++issued;
                        if (++s == RB) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                    ok = ok && !*abortFlag;
                }
                if (!ok) {
                    *abortFlag = 1;
                    for (uint32_t j = issued > RB ? issued - RB : 0; j < issued; ++j) mbar_wait(fullB(j % RB), (j / RB) & 1u);
                }
            }
        }
    } else if (warp == kEpiWarps + 1) {
        // MMA issuer: the whole warp runs the loop (uniform control flow and operands), one
        // elected lane issues
        const uint32_t leader = elect_one();
        const uint32_t idesc = idesc_bf16(sh.N, false, false);
        const uint32_t layout = layout_for_row_bytes(kRow);
        // descriptors advance by (byte offset >> 4) in their low 14-bit address field
        const uint64_t a0 = sdesc(base, 16, kHaloW * kRow, layout);
        const uint64_t b0 = sdesc(wBase, 16, 8 * kRow, layout);
        uint32_t sa0 = 0, phA = 0, sb = 0, phB = 0, it = 0;  // ring positions and their phases
        bool ok = true;
        if (kResident) ok = warp_wait(fullB(0), 0);
        for (uint32_t item = blockIdx.x; ok && item < items; item += gridDim.x, ++it) {
            const uint32_t buf = it & 1u, use = it >> 1;
            if (!(ok = warp_wait(accEmpty(buf), (use & 1u) ^ 1u))) break;
            // orders the MMAs after the epilogue's TMEM loads; the operands come from TMA and
            // need only their barriers
            tc_fence_after();
            const uint32_t acc = tmem + buf * sh.N;
            if constexpr (kResident && BLOCKS > 0) {
                uint64_t ad[BLOCKS];
#pragma unroll
                for (uint32_t g = 0; g < BLOCKS; ++g) {
                    const bool wrap = sa0 + g >= RA;
                    const uint32_t sa = wrap ? sa0 + g - RA : sa0 + g;
                    if (ok) ok = warp_wait(fullA(sa), phA ^ (wrap ? 1u : 0u));
                    ad[g] = a0 + sa * (kBlock >> 4);
                }
                if (!ok) break;
                const uint32_t ws = wSlice >> 4;
                if (leader) {
#pragma unroll
                    for (uint32_t tap = 0; tap < 9; ++tap) {
                        const uint32_t shift = ((tap / 3) * kHaloW + (tap % 3)) * (kRow >> 4);  // 16-byte units
#pragma unroll
                        for (uint32_t g = 0; g < BLOCKS; ++g) {
                            const uint64_t bd = b0 + (tap * BLOCKS + g) * ws;
#pragma unroll
                            for (uint32_t kk = 0; kk < CHUNK / 16; ++kk)
                                umma_bf16(acc, ad[g] + (shift + 2 * kk), bd + 2 * kk, idesc, (tap | g | kk) ? 1u : 0u);
                        }
                    }
#pragma unroll
                    for (uint32_t g = 0; g < BLOCKS; ++g) umma_commit(emptyA(sa0 + g >= RA ? sa0 + g - RA : sa0 + g));
                    umma_commit(accFull(buf));
                }
                __syncwarp();
            } else if constexpr (kByChunk) {
                if (leader) {
                    bool good = true;  // (once a wait gave up: garbage sums, the error flag, no more waits)
                    for (uint32_t g = 0; g < G; ++g) {
                        good = good && mbar_wait(fullA(sa0), phA);
#pragma unroll
                        for (uint32_t tap = 0; tap < 9; ++tap) {
                            const uint32_t shift = ((tap / 3) * kHaloW + (tap % 3)) * (kRow >> 4);
                            good = good && mbar_wait(fullB(sb), phB);
                            const uint64_t ad = a0 + (sa0 * (kBlock >> 4) + shift), bd = b0 + sb * (wSlice >> 4);
#pragma unroll
                            for (uint32_t kk = 0; kk < CHUNK / 16; ++kk)
                                umma_bf16(acc, ad + 2 * kk, bd + 2 * kk, idesc, (tap | g | kk) ? 1u : 0u);
                            umma_commit(emptyB(sb));
                            if (++sb == RB) {
                                sb = 0;
                                phB ^= 1u;
                            }
                        }
                        umma_commit(emptyA(sa0));
                        if (++sa0 == RA) {
                            sa0 = 0;
                            phA ^= 1u;
                        }
                    }
                    if (!good) *abortFlag = 1;
                    umma_commit(accFull(buf));
                }
                __syncwarp();
                ok = !warp_any(*abortFlag);
                continue;  // (the leader keeps the ring positions)
            } else {
                for (uint32_t g = 0; g < G && ok; ++g) {
                    const bool wrap = sa0 + g >= RA;
                    ok = warp_wait(fullA(wrap ? sa0 + g - RA : sa0 + g), phA ^ (wrap ? 1u : 0u));
                }
                if (!ok) break;
                // one lane runs the item's steps (a branch per step cost more than its MMAs)
                if (leader) {
#pragma unroll
                    for (uint32_t tap = 0; tap < 9; ++tap) {
                        const uint32_t shift = ((tap / 3) * kHaloW + (tap % 3)) * (kRow >> 4);
                        uint32_t sa = sa0;
                        for (uint32_t g = 0; g < G; ++g) {
                            // (a wait that gave up leaves garbage sums and the error flag)
                            if (!kResident && !mbar_wait(fullB(sb), phB)) *abortFlag = 1;
                            const uint64_t ad = a0 + (sa * (kBlock >> 4) + shift);
                            const uint64_t bd = b0 + (kResident ? tap * G + g : sb) * (wSlice >> 4);
#pragma unroll
                            for (uint32_t kk = 0; kk < CHUNK / 16; ++kk)
                                umma_bf16(acc, ad + 2 * kk, bd + 2 * kk, idesc, (tap | g | kk) ? 1u : 0u);
                            if (!kResident) {
                                umma_commit(emptyB(sb));
                                if (++sb == RB) {
                                    sb = 0;
                                    phB ^= 1u;
                                }
                            }
                            if (tap == 8) umma_commit(emptyA(sa));
                            if (++sa == RA) sa = 0;
                        }
                    }
                    umma_commit(accFull(buf));
                }
                __syncwarp();
                ok = !warp_any(*abortFlag);
            }
            sa0 += G;
            if (sa0 >= RA) {
                sa0 -= RA;
                phA ^= 1u;
            }
        }
        if (!ok) *abortFlag = 1;
        // every MMA has completed before TMEM is released
        if (leader) umma_commit(drain);
        __syncwarp();
        mbar_wait(drain, 0);
    } else {
        // Epilogue: lane l of a group's warp w owns tile row (pixel) 32w + l.  A warp's 32 rows
        // are four whole image rows of the tile, so it stages, pools and stores them by
        // itself: no barrier joins the warps.
        const uint32_t quad = warp & 3u, px = lane % kHTileW, py = lane / kHTileW;
        const uint32_t rowBytes = sh.stagingBytes / 128, sliceC = ep.outF32 ? rowBytes / 4 : rowBytes / 2;
        const uint32_t stg = sBase + warp * 32 * rowBytes;
        const uint32_t rowAddr = stg + lane * rowBytes, rowSwz = staged_unit(lane, 0, rowBytes) - lane * rowBytes;
        const bool plain = ep.bias && !ep.mask && !ep.outF32;  // bias, ReLU, bf16: the network's layers
        uint32_t it = 0;
        for (uint32_t item = blockIdx.x; item < items; item += gridDim.x, ++it) {
            const uint32_t buf = it & 1u, use = it >> 1;
            if (kEpiWarps == 8 && (warp >> 2) != buf) continue;  // the other group's buffer
            const TileAt ta = tile_at(sh, perImg, invImg, invX, item);
            const uint32_t n0 = ta.n0, b = ta.b, w0 = ta.w0, h0 = ta.h0 + quad * 4;  // the warp's rows
            const uint32_t h = h0 + py, w = w0 + px;
            const bool inside = h < sh.H;
            const size_t pix = ((size_t)b * sh.H + h) * sh.W + w;
            const size_t headAt = ((size_t)b * ep.headH + h) * ep.headW + w;
            float rgb[3] = {0.0f, 0.0f, 0.0f};  // (fetched ahead of the wait)
            if (ep.headDst && h < ep.headH && w < ep.headW)
                for (uint32_t j = 0; j < 3; ++j) rgb[j] = ep.headRgb[3 * headAt + j];
            if (warp_any(*abortFlag) || !warp_wait(accFull(buf), use & 1u)) {
                *abortFlag = 1;
                break;
            }
            __syncwarp();
            tc_fence_after();
            const uint32_t tAcc = tmem + ((quad * 32u) << 16) + buf * sh.N;
            if (ep.nOut) {
                for (uint32_t c0 = 0; c0 < sh.N; c0 += sliceC) {
                    if (lane == 0) bulk_wait_read<0>();  // the last store from this buffer has read it
                    __syncwarp();
                    if (sliceC % 32 == 0) {
                        for (uint32_t c = 0; c < sliceC; c += 32) {
                            uint32_t r[32];
                            tmem_ld32_async(tAcc + c0 + c, r);
                            tmem_ld_wait();
                            if (plain) {
                                stage32(rowAddr, rowSwz, c, biasS + n0 + c0 + c, ep.relu, r);
                            } else {
#pragma unroll
                                for (uint32_t q = 0; q < 2; ++q) {
                                    float v[16];
#pragma unroll
                                    for (uint32_t j = 0; j < 16; ++j) v[j] = __uint_as_float(r[16 * q + j]);
                                    finish16(ep, biasS, n0 + c0 + c + 16 * q, pix, inside, v);
                                    stage16(rowAddr, rowSwz, c + 16 * q, ep.outF32, v);
                                }
                            }
                        }
                    } else {
                        float v[16];  // sliceC == 16
                        tmem_ld16(tAcc + c0, v);
                        finish16(ep, biasS, n0 + c0, pix, inside, v);
                        stage16(rowAddr, rowSwz, 0, ep.outF32, v);
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0 && h0 < sh.H) {
                        for (uint32_t o = 0; o < ep.nOut; ++o)
                            tma_store_4d(&mo.m[o], stg, (int)(n0 + c0), (int)w0, (int)h0, (int)b);
                        bulk_commit();
                    }
                    if (ep.pool && h0 < sh.H) {
                        // 2x2 averages of the stored (bf16) values: one 8-channel group of one
                        // of the warp's 8 pooled pixels per step
                        const uint32_t lg = sliceC == 64 ? 3u : sliceC == 32 ? 2u : 1u;  // log2(sliceC / 8)
                        for (uint32_t k = lane; k < (8u << lg); k += 32) {
                            const uint32_t g8 = k & ((1u << lg) - 1u), q = k >> lg, qy = q / 4, qx = q % 4;
                            float s8[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
                            for (uint32_t d = 0; d < 4; ++d) {
                                const uint32_t r = (2 * qy + (d >> 1)) * kHTileW + 2 * qx + (d & 1u);
                                const uint4 u = ld_shared16(stg + staged_unit(r, g8, rowBytes));
                                const uint32_t ww[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                                for (uint32_t j = 0; j < 4; ++j) {
                                    const float2 f = __bfloat1622float2(*(const __nv_bfloat162*)&ww[j]);
                                    s8[2 * j] += f.x;
                                    s8[2 * j + 1] += f.y;
                                }
                            }
                            const size_t pp = ((size_t)b * (sh.H / 2) + h0 / 2 + qy) * (sh.W / 2) + w0 / 2 + qx;
                            *(uint4*)(ep.pool + pp * ep.poolStride + n0 + c0 + g8 * 8) =
                                make_uint4(bf2(s8[0] * 0.25f, s8[1] * 0.25f), bf2(s8[2] * 0.25f, s8[3] * 0.25f),
                                           bf2(s8[4] * 0.25f, s8[5] * 0.25f), bf2(s8[6] * 0.25f, s8[7] * 0.25f));
                        }
                    }
                }
            } else {
                for (uint32_t c0 = 0; c0 < sh.N; c0 += 16) {
                    float v[16];
                    tmem_ld16(tAcc + c0, v);
                    if (n0 + c0 < ep.coutValid && inside) {
                        finish16(ep, biasS, n0 + c0, pix, inside, v);
                        if (ep.headDst) {
                            // the network's last layer: radiance = expm1(log1p(rgb) + residual), cropped
                            if (h < ep.headH && w < ep.headW)
                                for (uint32_t j = 0; j < 3; ++j)
                                    ep.headDst[3 * headAt + j] = fmaxf(expm1f(log_radiance(rgb[j]) + v[j]), 0.0f);
                        } else {
                            store16(ep, pix * ep.outStride + n0 + c0, min(16u, ep.coutValid - n0 - c0), v);
                        }
                    }
                    __syncwarp();  // (the next load is .aligned)
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accEmpty(buf));
        }
        if (lane == 0) bulk_wait_all();
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abortFlag) atomicOr(err, 1u);
    __syncwarp();
    if (warp == 0) tmem_dealloc(tmem, sh.tmemCols);
}

// ---------------------------------------------------------------------------
// Weight gradient.  A block keeps the sums of one row of taps, or of all three (ROWS), of CB
// input and CA output channels in TMEM.  Per 8 x 16 pixel tile it loads G once and the
// input's halo once (10 pixels wide, 16 or 18 high); both are channel-contiguous (MN-major),
// K = pixels.  M holds the taps of a row times the input channels: the operand's channel
// groups are one pixel apart (LBO), so group dx reads the halo shifted by dx pixels (groups
// past the third are padding and not stored), and rows of 8 pixels are 10 halo rows apart as
// in k_conv_fwd.  N = the output channels, with an accumulator per dy.  Sums of a limited
// number of tiles are added in registers; then f32 atomics into dW, a warp's lanes along
// its input channels.
//
// kWide (CA = CB = 128): M is 128 input channels instead and a row's three taps are three
// accumulators, so M is full and N = 128 takes 94 cycles where two of 64 take 110-120; for wide
// layers over many pixels, which the MMAs bound (plan_wgrad): 512 -> 512 channels over 240 x 136
// pixels 196 us in blocks of 32 x 64 channels, 120 so; 161 with a block per tap.
//
// What bounds it: a block per tap loaded both operands nine times and padded M from the 16
// to 64 output channels of the wide layers to 128 (32 x 32 channels over 16 x 128 x 128
// pixels 63 us, 31 of them MMAs; L2 at 4.8 TB/s).  Now 14 us, 10 of them MMAs, the rest
// its start and its atomics; 192 -> 64 channels at half the width 37 -> 25 us, 256 -> 256 at
// an eighth 25 -> 15 us; a training pass at 16 x 128 x 128 1106 -> 846 us.

// The 4 x 4 transpose of four lanes' (lane & ~3 on) four values each.
__device__ __forceinline__ void transpose4(float* v, uint32_t lane) {
#pragma unroll
    for (uint32_t bit = 1; bit < 4; bit <<= 1) {
        const bool hi = lane & bit;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            if (k & bit) continue;
            const float got = __shfl_xor_sync(0xffffffffu, hi ? v[k] : v[k + bit], bit);
            if (hi) v[k] = got;
            else v[k + bit] = got;
        }
    }
}

template <int CA, int CB, int ROWS>
__global__ void __launch_bounds__(128, 1)
    k_conv_wgrad(const __grid_constant__ CUtensorMap mg, const __grid_constant__ CUtensorMap mx, WgradShape sh,
                  float* dW, uint32_t* err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr bool kWide = CB == 128;
    // channels are loaded in groups of at most 64, one after the other
    constexpr uint32_t kGroupsA = (CA + 63) / 64, kGroupsB = (CB + 63) / 64, kRowA = CA / kGroupsA * 2, kRowB = CB / kGroupsB * 2;
    constexpr uint32_t kHalo = wgrad_halo_rows(ROWS) * kHaloW, kHaloBytes = round_up(kHalo * kRowB, 1024), kGBytes = kTileP * kRowA;
    constexpr uint32_t kStage = kGroupsB * kHaloBytes + kGroupsA * kGBytes;
    constexpr uint32_t kCols = wgrad_cols(CA), kAccs = kWide ? 3 : ROWS;
    static_assert(kAccs * kCols <= (kWide ? 512 : ROWS == 1 ? 128 : 256), "the plan's TMEM columns");
    const uint32_t S = sh.stages;
    uint64_t* bars = (uint64_t*)(smem + S * kStage);
    uint32_t* tmemSlot = (uint32_t*)(bars + 2 * S + 1);
    volatile uint32_t* abortFlag = tmemSlot + 1;
    const uint32_t base = smem_u32(smem);
    auto full = [&](uint32_t s) { return smem_u32(bars + s); };
    auto empty = [&](uint32_t s) { return smem_u32(bars + S + s); };
    const uint32_t accum = smem_u32(bars + 2 * S);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t ci0 = blockIdx.y * CB, co0 = blockIdx.z / (3 / ROWS) * CA;
    const uint32_t dy0 = blockIdx.z % (3 / ROWS);  // the block's first row of taps
    const uint32_t t0 = blockIdx.x * sh.tilesPerCta, t1 = min(sh.tilesTotal, t0 + sh.tilesPerCta);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < S; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(accum, 1);
        *abortFlag = 0;
        fence_mbar_init();
        prefetch_map(&mg);
        prefetch_map(&mx);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmemSlot), sh.tmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmemSlot;
    grid_launch_dependents();
    grid_wait();
    const uint32_t perImg = sh.tilesX * sh.tilesY;
    const uint32_t kSteps = t1 > t0 ? t1 - t0 : 0;
    const uint32_t idesc = idesc_bf16(CA, true, true);
    const uint32_t layG = layout_for_row_bytes(kRowA), layX = layout_for_row_bytes(kRowB);
    const bool leader = warp < 2 && elect_one();
    uint32_t issued = 0, s = 0, ph = warp == 0 ? 1 : 0;  // the loading or the MMA warp's place in the ring

    // The block's tiles in sums of at most sh.sumTiles in TMEM (see plan_wgrad), which meet in
    // registers: row (warp, lane), columns dy * CA + co.
    const uint32_t rows = tmem + ((warp * 32u) << 16);  // this warp's rows of the accumulators
    float total[kWide ? 1 : ROWS * CA] = {};
    bool ok = true;
    for (uint32_t k0 = 0, sum = 0; ok && k0 < kSteps; k0 += sh.sumTiles, ++sum) {
        const uint32_t k1 = min(kSteps, k0 + sh.sumTiles);
        if (warp == 0) {
            if (leader) {
                // (the next sum's first tiles load while this one is read)
                for (const uint32_t upTo = min(kSteps, k1 + S); issued < upTo; ++issued) {
                    if (!mbar_wait(empty(s), ph)) {
                        *abortFlag = 1;
                        break;
                    }
                    const uint32_t t = t0 + issued;
                    const uint32_t b = t / perImg, rem = t % perImg;
                    const int h0 = (int)((rem / sh.tilesX) * kHTileH), w0 = (int)((rem % sh.tilesX) * kHTileW);
                    mbar_expect_tx(full(s), kGroupsB * kHalo * kRowB + kGroupsA * kGBytes);
                    const uint32_t sa = base + s * kStage;
#pragma unroll
                    for (uint32_t g = 0; g < kGroupsB; ++g)
                        tma_load_4d(sa + g * kHaloBytes, &mx, full(s), (int)(ci0 + 64 * g), w0 - 1, h0 - 1 + (int)dy0, (int)b);
#pragma unroll
                    for (uint32_t g = 0; g < kGroupsA; ++g)
                        tma_load_4d(sa + kGroupsB * kHaloBytes + g * kGBytes, &mg, full(s), (int)(co0 + 64 * g), w0, h0, (int)b);
                    if (++s == S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
        } else if (warp == 1) {
            for (uint32_t k = k0; k < k1; ++k) {
                if (!warp_wait(full(s), ph)) {
                    *abortFlag = 1;
                    break;
                }
                const uint32_t b0 = base + s * kStage;
                const uint64_t xd = sdesc(b0, kWide ? kHaloBytes : kRowB, kHaloW * kRowB, layX);
                const uint64_t gd = sdesc(b0 + kGroupsB * kHaloBytes, kGroupsA > 1 ? kGBytes : 0, 8 * kRowA, layG);
                if (leader) {
#pragma unroll
                    for (uint32_t kk = 0; kk < kTileP / 16; ++kk)
#pragma unroll
                        for (uint32_t a = 0; a < kAccs; ++a)  // 16 pixels: two rows of the tile; a: dy, or dx of kWide
                            umma_bf16(tmem + a * kCols,
                                      xd + ((2 * kk + (kWide ? 0 : a)) * kHaloW + (kWide ? a : 0)) * (kRowB / 16),
                                      gd + kk * kRowA, idesc, (k - k0 | kk) ? 1u : 0u);
                    umma_commit(empty(s));
                }
                __syncwarp();
                if (++s == S) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (leader) umma_commit(accum);
        }
        __syncwarp();

        const bool ready = warp_wait(accum, sum & 1u) && !warp_any(*abortFlag);
        tc_fence_after();
        if (!ready) {
            if (lane == 0) atomicOr(err, 1u);
        } else if constexpr (!kWide) {
            // one of several sums: added to the others, which the last one leaves in its columns
            if (warp * 32 < 3 * CB && sh.sumTiles < sh.tilesPerCta) {
#pragma unroll
                for (uint32_t j = 0; j < ROWS * CA / 16; ++j) {
                    float v[16];
                    tmem_ld16(rows + j / (CA / 16) * kCols + j % (CA / 16) * 16, v);
#pragma unroll
                    for (uint32_t i = 0; i < 16; ++i) total[16 * j + i] += v[i];
                }
                if (k1 == kSteps) {
#pragma unroll
                    for (uint32_t j = 0; j < ROWS * CA / 16; ++j)
                        tmem_st16(rows + j / (CA / 16) * kCols + j % (CA / 16) * 16, total + 16 * j);
                    tmem_st_wait();
                }
            }
        }
        tc_fence_before();
        ok = !__syncthreads_or(!ready);
        tc_fence_after();
    }
    if (ok && kSteps > 0 && warp * 32 < 3 * CB) {
        // row dx * CB + ci, column co, of accumulator dy (kWide: row ci of accumulator dx); a
        // short loop: unrolled over registers it ran from cold instruction memory, 2.4 us
        const uint32_t row = warp * 32 + lane, rowDx = row / CB, ci = ci0 + row % CB;
        const bool vec = ((uintptr_t)dW & 15u) == 0, mine = rowDx < 3 && ci < sh.Cin;
#pragma unroll 1
        for (uint32_t j = 0; j < kAccs * CA / 16; ++j) {
            const uint32_t acc = j / (CA / 16), c0 = j % (CA / 16) * 16, co = co0 + c0;
            const uint32_t tap = kWide ? dy0 * 3 + acc : (dy0 + acc) * 3 + rowDx;
            float v[16];
            tmem_ld16(rows + acc * kCols + c0, v);
            if (vec) {
                // four lanes' inputs of one output channel meet in a lane, an atomic per 16 bytes:
                // 64 -> 64 channels over 16 x 8 pixels 10.1 -> 8.3 us, a training pass of
                // 16 x 128 x 128 862 -> 846
#pragma unroll
                for (uint32_t i = 0; i < 16; i += 4) {
                    transpose4(v + i, lane);
                    const uint32_t c = co + i + (lane & 3u);
                    if (mine && c < sh.coutStore)
                        atomicAdd((float4*)(dW + ((size_t)c * 9 + tap) * sh.Cin + (ci & ~3u)),
                                  make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
                }
            } else if (mine) {
                float* o = dW + ((size_t)co * 9 + tap) * sh.Cin + ci;
#pragma unroll
                for (uint32_t i = 0; i < 16; ++i)
                    if (co + i < sh.coutStore) atomicAdd(o + (size_t)i * 9 * sh.Cin, v[i]);
            }
            __syncwarp();  // (the next load is .aligned)
        }
    }
    // a block that gave up lets its copies in flight land first (bounded)
    if (warp == 0 && leader) {
        if (*abortFlag) {
            for (uint32_t k = issued > S ? issued - S : 0; k < issued; ++k) mbar_wait(full(k % S), (k / S) & 1u);
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, sh.tmemCols);
}

// ---------------------------------------------------------------------------
// host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

static CUtensorMapSwizzle swizzle_for(uint32_t rowBytes) {
    return rowBytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                           : rowBytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

static uint32_t pow2_cols(uint32_t n) {
    uint32_t c = 32;
    while (c < n) c <<= 1;
    return c;
}

// Dynamic shared memory that keeps (blocks per SM) x (TMEM columns) within the 512
// columns of an SM: the allocation of a block that does not fit would wait.
static uint32_t smem_for(uint32_t need, uint32_t tmemCols) {
    const uint32_t smPool = 228 * 1024, perBlockReserve = 1024;
    uint32_t maxBlocks = std::max(1u, 512u / tmemCols);
    uint32_t s = need;
    while (smPool / (s + perBlockReserve) > maxBlocks) s += 1024;
    return s;
}

int chunk_for(uint32_t c) { return c % 64 == 0 ? 64 : c % 32 == 0 ? 32 : 16; }

// Work split and rings of a forward launch.  Weights stay resident when they take at most
// 72 KB (two blocks then share an SM where their rings fit); otherwise they stream, and
// where an image has fewer tiles than the GPU has SMs the output channels are split over
// blocks (a tile of 256 -> 256 channels takes a block 15 us per 128 output channels).
int plan_fwd(uint32_t B, uint32_t H, uint32_t W, uint32_t Cin, uint32_t N, bool outF32, uint32_t numSMs, FwdPlan* p) {
    if (Cin == 0 || Cin % 16 || N == 0 || N % 16 || W % 8 || H % 8 || B == 0) return 1;
    FwdShape& sh = p->shape;
    sh.B = B;
    sh.H = H;
    sh.W = W;
    sh.Cin = Cin;
    sh.tilesX = W / kHTileW;
    sh.tilesY = (H + kHTileH - 1) / kHTileH;
    p->chunk = chunk_for(Cin);
    const uint32_t kRow = p->chunk * 2, G = Cin / p->chunk, block = halo_block_bytes(p->chunk);
    const uint32_t tiles = B * sh.tilesX * sh.tilesY;
    sh.nSplit = 1;
    p->resident = N <= 128 && 9 * Cin * N * 2 <= 72u * 1024u;
    p->byChunk = false;
    if (!p->resident) {
        // at most 192 channels an item, so that the weight ring holds several slices, where
        // that takes four items at most; otherwise as few as an MMA's 256 channels allow
        auto fits = [&](uint32_t most) { return N / sh.nSplit <= most && N % (16 * sh.nSplit) == 0; };
        while (sh.nSplit <= 4 && !fits(192)) ++sh.nSplit;
        if (!fits(192))
            for (sh.nSplit = 1; !fits(256);)
                if (++sh.nSplit > N / 16) return 1;
        while (tiles * sh.nSplit * 2 <= numSMs && (N / sh.nSplit) % 64 == 0) sh.nSplit *= 2;
    }
    sh.N = N / sh.nSplit;
    sh.tmemCols = pow2_cols(2 * sh.N);  // double-buffered accumulator
    const uint32_t wSlice = sh.N * kRow, sliceC = outF32 ? (sh.N % 32 ? 16u : 32u) : (sh.N % 64 == 0 ? 64u : sh.N % 32 == 0 ? 32u : 16u);
    p->sliceC = sliceC;
    sh.stagingBytes = 128 * sliceC * (outF32 ? 4 : 2);
    const uint32_t staging = sh.stagingBytes * (fwd_epilogue_warps(p->resident) / 4);
    const uint32_t fixed = staging + 1024 /* bias */ + 1024 /* alignment */ + 1024 /* barriers */;
    auto need = [&](uint32_t ra, uint32_t rb) {
        return ra * block + round_up((p->resident ? 9 * G : rb) * wSlice, 1024) + fixed;
    };
    const uint32_t limit = 227u * 1024u, smPool = 228u * 1024u;
    if (p->resident) {
        // two blocks per SM where that leaves each three items' halos in flight
        sh.stagesB = 1;
        sh.stagesA = G;
        for (uint32_t blocks = std::min(2u, 512u / sh.tmemCols); blocks >= 1; --blocks) {
            const uint32_t room = std::min(limit, smPool / blocks - 1024u);
            uint32_t ra = 8 * G;
            while (ra > G && need(ra, 1) > room) --ra;
            if (blocks == 1 || (need(ra, 1) <= room && ra >= 3 * G)) {
                sh.stagesA = ra;
                break;
            }
        }
    } else {
        // halos of one item at least and of two if that leaves six weight slices (a slice is
        // 200-400 cycles of MMAs and takes ~2000 to be released and arrive)
        sh.stagesA = 2 * G;
        while (sh.stagesA > G && need(sh.stagesA, 6) > limit) --sh.stagesA;
        sh.stagesB = 16;
        while (sh.stagesB > 2 && need(sh.stagesA, sh.stagesB) > limit) --sh.stagesB;
        // Chunk by chunk where the halos leave room for fewer than sixteen MMAs' weights (more
        // than 384 channels): the MMAs waited for their slices otherwise (16 x 128 x 128
        // 448 -> 192 260 us by chunk; with one slice beside seven chunks no plan at all), and
        // inputs whose chunks do not fit are held no other way (512 -> 128 at 1920 x 1088 1690
        // us).  And with 16- and 32-channel chunks, one or two MMAs a slice: the straight loop
        // over nine taps steps twice as fast as the one over chunks (144 -> 32 at 960 x 544 361
        // us tap by tap, 190 by chunk; 96 -> 96 150, 131).
        const uint32_t mmas = p->chunk / 16;
        p->byChunk = p->chunk < 64 || need(sh.stagesA, sh.stagesB) > limit || sh.stagesB * mmas < 16;
        if (p->byChunk) {
            sh.stagesA = std::min(G, 4u);
            while (sh.stagesA > 2 && need(sh.stagesA, 16 / mmas) > limit) --sh.stagesA;
            sh.stagesB = 16;
            while (sh.stagesB > 2 && need(sh.stagesA, sh.stagesB) > limit) --sh.stagesB;
        }
    }
    if (need(sh.stagesA, sh.stagesB) > limit) return 1;
    p->smem = smem_for(need(sh.stagesA, sh.stagesB), sh.tmemCols);
    const uint32_t perSM = std::max(1u, std::min(228u * 1024u / (p->smem + 1024u), 512u / sh.tmemCols));
    p->grid = std::min(tiles * sh.nSplit, perSM * numSMs);
    return 0;
}

static int encode4(CUtensorMap* m, CUtensorMapDataType type, const void* base, const cuuint64_t (&dims)[4],
                   const cuuint64_t (&strides)[3], const cuuint32_t (&box)[4], uint32_t rowBytes) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return 1;
    if (((uintptr_t)base & 15u) || strides[0] % 16 || strides[1] % 16 || strides[2] % 16) return 2;
    const cuuint32_t es[4] = {1, 1, 1, 1};
    CUresult r = enc(m, type, 4, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     swizzle_for(rowBytes), CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 3;
}

int make_input_map(const FwdPlan& p, const void* x, CUtensorMap* mx) {
    const FwdShape& sh = p.shape;
    const cuuint64_t px = (cuuint64_t)sh.Cin * 2;
    return encode4(mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, {sh.Cin, sh.W, sh.H, sh.B}, {px, px * sh.W, px * sh.W * sh.H},
                   {(cuuint32_t)p.chunk, kHaloW, kHaloH, 1}, p.chunk * 2);
}

int make_weight_map(const FwdPlan& p, const void* w, CUtensorMap* mw) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return 1;
    const FwdShape& sh = p.shape;
    if ((uintptr_t)w & 15u) return 2;
    const cuuint64_t dims[2] = {9ull * sh.Cin, (cuuint64_t)sh.N * sh.nSplit};
    const cuuint64_t strides[1] = {18ull * sh.Cin};
    const cuuint32_t box[2] = {(cuuint32_t)p.chunk, sh.N};
    const cuuint32_t es[2] = {1, 1};
    CUresult r = enc(mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(w), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(p.chunk * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 3;
}

int make_out_maps(const FwdPlan& p, void* out, uint32_t C, uint32_t stride, uint32_t offset, bool f32, bool up, OutMaps* mo) {
    const FwdShape& sh = p.shape;
    const size_t es = f32 ? 4 : 2;
    const uint32_t f = up ? 2 : 1;
    memset(mo, 0, sizeof(*mo));
    for (uint32_t o = 0; o < (up ? 4u : 1u); ++o) {
        const size_t px = stride * es, row = px * sh.W * f;
        uint8_t* base = (uint8_t*)out + offset * es + (o >> 1) * row + (o & 1u) * px;
        const int rc = encode4(&mo->m[o], f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base,
                               {C, sh.W, sh.H, sh.B}, {px * f, row * f, row * f * sh.H},
                               {p.sliceC, kHTileW, 4, 1}, (uint32_t)(p.sliceC * es));
        if (rc) return rc;
    }
    return 0;
}

int make_wgrad_maps(const WgradPlan& p, const void* g, const void* x, uint32_t B, uint32_t H, uint32_t W, uint32_t Cin,
                    uint32_t Cout, CUtensorMap* mg, CUtensorMap* mx) {
    auto nhwc = [&](CUtensorMap* m, const void* base, uint32_t C, uint32_t boxC, uint32_t boxW, uint32_t boxH) {
        return encode4(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, {C, W, H, B},
                       {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2}, {boxC, boxW, boxH, 1},
                       boxC * 2);
    };
    const int rc = nhwc(mg, g, Cout, std::min(64u, p.ca), kHTileW, kHTileH);
    return rc ? rc : nhwc(mx, x, Cin, std::min(64u, p.cb), kHaloW, wgrad_halo_rows(p.rows));
}

int plan_wgrad(uint32_t B, uint32_t H, uint32_t W, uint32_t Cin, uint32_t Cout, uint32_t numSMs, WgradPlan* p) {
    if (Cin == 0 || Cin % 16 || Cout == 0 || Cout % 16 || W % 16 || H % 8 || B == 0) return 1;
    if (Cin > 512 || (Cin > 256 && Cin % 32)) return 1;
    WgradShape& sh = p->shape;
    sh.Cin = Cin;
    sh.coutStore = Cout;
    sh.tilesX = W / kHTileW;
    sh.tilesY = (H + kHTileH - 1) / kHTileH;
    sh.tilesTotal = B * sh.tilesX * sh.tilesY;
    // Widths by what fills an MMA, not by what divides the channels: it takes the same time up
    // to N = 64, and M holds three taps of 32 input channels; channels past the last are loaded
    // as zeros and not stored (240 -> 240 over 4 x 64 x 64 in blocks of 16 x 16 171 us, here 34).
    p->ca = Cout <= 16 ? 16 : Cout <= 32 ? 32 : 64;
    p->cb = Cin <= 16 ? 16 : 32;
    // The longest sum in TMEM, where every step is cut to f32, so that the error grows with the
    // length: the tiles that two blocks an SM, of one tap, 128 output and 256 input channels
    // each, would have (256 -> 256 channels over 16 x 16 x 16 pixels: 4.5e-7 from 64-bit sums
    // with 4 tiles in one sum, 2.3e-7 with 2).
    const uint32_t cells = 9 * ((Cin + 255) / 256) * ((Cout + 127) / 128);
    const uint32_t parts = std::min((2 * numSMs + cells - 1) / cells, sh.tilesTotal);
    const uint32_t longest = (sh.tilesTotal + parts - 1) / parts;
    // One wave of blocks, two an SM: one covers the other's start and atomics (one an SM:
    // 36 us for 96 -> 32 channels at full width, 32 with two), and a second wave would cost
    // a start (256 -> 256 channels at an eighth: 17 us, 24 with twice the blocks).  The
    // full-width layers (up to 32 output channels, the most pixels) give each row of taps
    // its own blocks: a third of the splits' atomics for G loaded three times (a training
    // pass 862 -> 850 us); with several blocks of input channels their splits would be so
    // few that a block's sums in TMEM, which truncate, grow longer than they were, so four
    // blocks share an SM there.  So do narrow gradients of a few tiles, whose blocks of all
    // taps would leave SMs idle (64 -> 64 channels over 16 x 8 pixels 8.3 us, 5.0 with a row
    // a block).
    const uint32_t ciBlocks = (Cin + p->cb - 1) / p->cb;
    p->rows = p->ca == 64 && ciBlocks * ((Cout + 63) / 64) * sh.tilesTotal >= numSMs ? 3 : 1;
    const uint32_t coBlocks = (Cout + p->ca - 1) / p->ca * (3 / p->rows);
    const uint32_t perSM = p->rows == 1 && ciBlocks > 1 ? 4 : 2;
    sh.tmemCols = 512 / perSM;  // of which rows * wgrad_cols(ca) are used: 192 of 256, or 32 or 64
    const uint32_t stage = round_up(wgrad_halo_rows(p->rows) * kHaloW * p->cb * 2, 1024) + kTileP * p->ca * 2;
    sh.stages = std::min(6u, (224u * 1024u / perSM - 2048u) / stage);
    p->smem = smem_for(sh.stages * stage + (2 * sh.stages + 1) * 8 + 16 + 1024, sh.tmemCols);
    uint32_t splits = std::min(std::max(1u, perSM * numSMs / (ciBlocks * coBlocks)), sh.tilesTotal);
    sh.tilesPerCta = (sh.tilesTotal + splits - 1) / splits;
    splits = (sh.tilesTotal + sh.tilesPerCta - 1) / sh.tilesPerCta;
    p->grid = dim3(splits, ciBlocks, coBlocks);
    // A block of more tiles than the longest sum reads several and adds them in registers: more
    // blocks would each add all their weights to memory (a training pass of 16 x 128 x 128 858 us
    // without the limit, 862 with it, 874 with blocks of that length).
    const uint32_t sums = (sh.tilesPerCta + longest - 1) / longest;
    sh.sumTiles = (sh.tilesPerCta + sums - 1) / sums;
    if (Cin <= 64 || Cout <= 64) return 0;

    // kWide, one block an SM, with the splits (no longer sums) that take the least time in whole
    // waves, where that beats the blocks above.  Measured on 148 SMs: a tile 1.17 us, a block's
    // start and atomics as much as seven tiles, and 5 us; above 1.4 us a tile (of two blocks an SM) and
    // 9 us.  512 -> 512 over 240 x 136 pixels 196 us above, 120 kWide, over 64 x 64 34 and 36;
    // 256 -> 256 over 480 x 272 167 and 117, over 64 x 64 15 and 27.
    const uint32_t ciWide = (Cin + 127) / 128, coWide = (Cout + 127) / 128 * 3;
    uint32_t waves = ~0u, each = 0;
    for (uint32_t n = parts; n <= std::min(sh.tilesTotal, 8 * parts); ++n) {
        const uint32_t tiles = (sh.tilesTotal + n - 1) / n, time = (n * ciWide * coWide + numSMs - 1) / numSMs * (tiles + 7);
        if (time < waves) {
            waves = time;
            each = tiles;
        }
    }
    if (1.17f * waves + 5.0f < 1.4f * sh.tilesPerCta + 9.0f) {
        p->ca = p->cb = 128;
        p->rows = 1;
        sh.tilesPerCta = sh.sumTiles = each;
        p->grid = dim3((sh.tilesTotal + each - 1) / each, ciWide, coWide);
        sh.tmemCols = 512;
        sh.stages = 3;
        const uint32_t wide = 2 * (round_up(wgrad_halo_rows(1) * kHaloW * 128, 1024) + kTileP * 128);
        p->smem = smem_for(sh.stages * wide + (2 * sh.stages + 1) * 8 + 16 + 1024, sh.tmemCols);
    }
    return 0;
}

template <class K>
static cudaError_t set_smem(K kern, uint32_t bytes) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

cudaError_t launch_fwd(const FwdPlan& p, const CUtensorMap& mx, const CUtensorMap& mw, const OutMaps& mo,
                       const Epilogue& ep, bool overlap, uint32_t* err, cudaStream_t st) {
    cudaError_t e = cudaErrorInvalidValue;
    // overlap: launched while its predecessor drains (see the kernel's grid_wait), so that its
    // barriers, TMEM and resident weights are ready when the predecessor ends (300 x 170
    // frame 226 -> 180 us)
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(p.grid);
    lc.blockDim = dim3(fwd_threads(p.resident));
    lc.dynamicSmemBytes = p.smem;
    lc.stream = st;
    lc.attrs = &at;
    lc.numAttrs = overlap ? 1 : 0;
#define WRK_FWD_CASE(CHUNK, RES, BLOCKS, BY)                                                                               \
    if (p.chunk == CHUNK && p.resident == RES && p.byChunk == BY && (BLOCKS == 0 || p.shape.Cin == CHUNK * BLOCKS)) {      \
        e = set_smem(k_conv_fwd<CHUNK, RES, BLOCKS, BY>, p.smem);                                                          \
        if (e == cudaSuccess)                                                                                              \
            e = cudaLaunchKernelEx(&lc, k_conv_fwd<CHUNK, RES, BLOCKS, BY>, mx, mw, mo, p.shape, ep, err);                 \
        return e != cudaSuccess ? e : cudaGetLastError();                                                                  \
    }
    WRK_FWD_CASE(16, true, 1, false)
    WRK_FWD_CASE(32, true, 1, false)
    WRK_FWD_CASE(32, true, 3, false)
    WRK_FWD_CASE(64, true, 1, false)
    WRK_FWD_CASE(16, true, 0, false)
    WRK_FWD_CASE(32, true, 0, false)
    WRK_FWD_CASE(64, true, 0, false)
    WRK_FWD_CASE(16, false, 0, false)
    WRK_FWD_CASE(32, false, 0, false)
    WRK_FWD_CASE(64, false, 0, false)
    WRK_FWD_CASE(16, false, 0, true)
    WRK_FWD_CASE(32, false, 0, true)
    WRK_FWD_CASE(64, false, 0, true)
#undef WRK_FWD_CASE
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_wgrad(const WgradPlan& p, const CUtensorMap& mg, const CUtensorMap& mx, float* dW, bool overlap,
                         uint32_t* err, cudaStream_t st) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = p.grid;
    lc.blockDim = dim3(128);
    lc.dynamicSmemBytes = p.smem;
    lc.stream = st;
    lc.attrs = &at;
    lc.numAttrs = overlap ? 1 : 0;
    cudaError_t e = cudaSuccess;
#define WRK_WGRAD_CASE(A, B, ROWS)                                                           \
    if (p.ca == A && p.cb == B && p.rows == ROWS) {                                          \
        e = set_smem(k_conv_wgrad<A, B, ROWS>, p.smem);                                      \
        if (e == cudaSuccess)                                                                \
            e = cudaLaunchKernelEx(&lc, k_conv_wgrad<A, B, ROWS>, mg, mx, p.shape, dW, err); \
        return e != cudaSuccess ? e : cudaGetLastError();                                    \
    }
    WRK_WGRAD_CASE(128, 128, 1)
    WRK_WGRAD_CASE(64, 32, 3)
    WRK_WGRAD_CASE(64, 16, 3)
    WRK_WGRAD_CASE(64, 32, 1)
    WRK_WGRAD_CASE(64, 16, 1)
    WRK_WGRAD_CASE(32, 32, 1)
    WRK_WGRAD_CASE(32, 16, 1)
    WRK_WGRAD_CASE(16, 32, 1)
    WRK_WGRAD_CASE(16, 16, 1)
#undef WRK_WGRAD_CASE
    return cudaErrorInvalidValue;
}

}  // namespace conv
}  // namespace wrk
