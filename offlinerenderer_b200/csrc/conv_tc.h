// Host interface of the tcgen05 convolution kernels (conv_tc.cu).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace wrk {
namespace conv {

struct FwdShape {
    uint32_t B, H, W, Cin;
    uint32_t N, nSplit;       // output channels of one work item (a multiple of 16, <= 256); items per tile
    uint32_t tilesX, tilesY;  // 8 x 16 pixel tiles (the last row of tiles may overhang the image)
    uint32_t stagesA, stagesB;  // ring slots: halo chunks, weight slices
    uint32_t stagingBytes;      // one staged output slice (the epilogue warps' 4 x 32 pixels)
    uint32_t tmemCols;
};

// What the forward kernel does with the accumulator of output channel co:
// (+ bias[co]) -> (ReLU) -> (x 0 where mask <= 0) -> store.  nOut > 0: by TMA through the
// launch's output maps (bf16 or f32; four maps = the 2x nearest upsample), and the 2x2
// average of the stored bf16 values into `pool` when it is set.  nOut = 0: the cropped
// output image when headDst is set, else plain stores to out[pixel*outStride + co] for
// co < coutValid.
struct Epilogue {
    const float* bias;  // bias[co] added for co < nBias (f32, at most 256 channels)
    uint32_t nBias;
    uint32_t nOut;
    void* out;
    uint32_t outStride, coutValid;
    uint32_t relu, outF32;
    const __nv_bfloat16* mask;
    uint32_t maskStride;
    __nv_bfloat16* pool;  // [B][H/2][W/2][poolStride]
    uint32_t poolStride;
    const float* headRgb;  // [B][headH][headW][3]
    float* headDst;
    uint32_t headH, headW;
};

struct WgradShape {
    uint32_t Cin;
    uint32_t coutStore;  // rows of dW that exist (<= the channels of G)
    uint32_t tilesX, tilesY, tilesTotal, tilesPerCta;
    uint32_t sumTiles;    // tiles of one sum in TMEM
    uint32_t stages, tmemCols;
};

// Output tensor maps of a forward launch: one, or one per child pixel of an upsample.
struct OutMaps {
    CUtensorMap m[4];
};
struct FwdPlan {
    FwdShape shape;
    int chunk;        // input channels per halo chunk
    uint32_t sliceC;  // output channels per staged slice
    uint32_t smem, grid;
    bool resident;    // the whole weight tensor stays in shared memory
    bool byChunk;     // streamed weights: an item runs chunk by chunk (its chunks do not fit together)
};
struct WgradPlan {
    WgradShape shape;
    uint32_t ca, cb, rows, smem;  // output channels, input channels and rows of taps of a block
    dim3 grid;
};

int chunk_for(uint32_t channels);
// All map functions return 0 on success.
// Maps of a weight gradient: G and the layer's input, NHWC bf16.
int make_wgrad_maps(const WgradPlan& p, const void* g, const void* x, uint32_t B, uint32_t H, uint32_t W, uint32_t Cin,
                    uint32_t Cout, CUtensorMap* mg, CUtensorMap* mx);
int plan_fwd(uint32_t B, uint32_t H, uint32_t W, uint32_t Cin, uint32_t N, bool outF32, uint32_t numSMs, FwdPlan* p);
int plan_wgrad(uint32_t B, uint32_t H, uint32_t W, uint32_t Cin, uint32_t Cout, uint32_t numSMs, WgradPlan* p);
// Tensor maps of a forward plan: the input, the weights [N * nSplit][9 * Cin] bf16, and
// the output (its first C channels, from channel `offset` on of a buffer `stride` channels
// wide; up = the 2x nearest upsample of the output, whose buffer is 2W x 2H).
int make_input_map(const FwdPlan& p, const void* x, CUtensorMap* mx);
int make_weight_map(const FwdPlan& p, const void* w, CUtensorMap* mw);
int make_out_maps(const FwdPlan& p, void* out, uint32_t C, uint32_t stride, uint32_t offset, bool f32, bool up, OutMaps* mo);
// overlap: the launch may begin before the stream's previous kernel has ended; the weights
// and the bias must then be older than that kernel.
cudaError_t launch_fwd(const FwdPlan& p, const CUtensorMap& mx, const CUtensorMap& mw, const OutMaps& mo,
                       const Epilogue& ep, bool overlap, uint32_t* err, cudaStream_t st);
cudaError_t launch_wgrad(const WgradPlan& p, const CUtensorMap& mg, const CUtensorMap& mx, float* dW, bool overlap,
                         uint32_t* err, cudaStream_t st);

}  // namespace conv
}  // namespace wrk
