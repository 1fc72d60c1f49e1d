// Plans of the 3x3 convolution and of its weight gradient for every channel count the entry
// points take, without a GPU: one line "Cin Cout f32 H W B rc" (f32 = 2: weight gradient) per
// plan that is refused or that does not hold together.
// Built and run by tests/test_conv_plans.py.
#include <algorithm>
#include <cstdio>

#include "conv_tc.h"

using namespace wrk::conv;

int main() {
    const uint32_t sizes[][3] = {{1, 8, 16}, {1, 64, 128}, {1, 1088, 1920}, {16, 128, 128}};
    long plans = 0, byChunk = 0, wide = 0;
    for (uint32_t cin = 16; cin <= 2048; cin += 16)
        for (uint32_t n = 16; n <= 256; n += 16)
            for (int f32 = 0; f32 < 2; ++f32)
                for (auto& z : sizes) {
                    FwdPlan p{};
                    const int rc = plan_fwd(z[0], z[1], z[2], cin, n, f32 != 0, 148, &p);
                    const FwdShape& s = p.shape;
                    const uint32_t chunks = rc ? 0 : cin / p.chunk;
                    const bool ok =
                        rc == 0 && cin % p.chunk == 0 && s.N * s.nSplit == n && s.N % 16 == 0 && s.N <= 256 && s.N % p.sliceC == 0 &&
                        s.tmemCols >= 2 * s.N && s.tmemCols <= 512 && p.smem <= 227 * 1024 && p.grid > 0 &&
                        (2 * s.stagesA + 2 * s.stagesB + 5) * 8 + 8 <= 1024 &&  // the barriers' share
                        // all chunks of an item at once unless it runs chunk by chunk, and a ring of weights
                        // (split further only where an image has few tiles)
                        (s.nSplit <= 4 || z[1] < 128) &&
                        (p.byChunk ? s.stagesA >= 2 || s.stagesA == chunks : s.stagesA >= chunks) &&
                        // (a slice of fewer than four MMAs is worth its wait only in the loop by chunk)
                        (p.resident ? !p.byChunk : s.stagesB >= 2 && (p.chunk == 64 || p.byChunk));
                    ++plans;
                    byChunk += p.byChunk;
                    if (!ok) std::printf("%u %u %d %u %u %u %d\n", cin, n, f32, z[1], z[2], z[0], rc);
                }
    for (uint32_t cin = 16; cin <= 512; cin += cin < 256 ? 16 : 32)
        for (uint32_t cout = 16; cout <= 512; cout += 16)
            for (auto& z : sizes) {
                WgradPlan p{};
                const int rc = plan_wgrad(z[0], z[1], z[2], cin, cout, 148, &p);
                const WgradShape& s = p.shape;
                const uint32_t tiles = z[0] * (z[2] / 8) * ((z[1] + 15) / 16);
                // the longest sum a tensor-memory accumulator may take: the tiles that two
                // blocks per SM of one tap, 128 output and 256 input channels each, would share
                const uint32_t cells = 9 * ((cin + 255) / 256) * ((cout + 127) / 128);
                const uint32_t parts = std::min((2 * 148 + cells - 1) / cells, tiles);
                const bool ok = rc == 0 && s.tilesTotal == tiles && p.grid.x * s.tilesPerCta >= tiles &&
                                (p.grid.x - 1) * s.tilesPerCta < tiles && p.grid.y * p.cb >= cin &&
                                p.grid.z * p.rows / 3 * p.ca >= cout && p.smem <= 227 * 1024 && s.stages >= 2 &&
                                (p.ca == 128 ? 3 : p.rows) * ((p.ca + 31) / 32 * 32) <= s.tmemCols && s.sumTiles > 0 &&
                                s.sumTiles <= (tiles + parts - 1) / parts &&
                                (p.ca == 128 ? p.cb == 128 && p.rows == 1 && s.sumTiles == s.tilesPerCta && cin > 64 && cout > 64
                                             // no more blocks of channels than an MMA's rows and columns call for
                                             : p.grid.y == (cin + 31) / 32 &&
                                                   p.grid.z * p.rows / 3 == (cout <= 32 ? 1 : (cout + 63) / 64) &&
                                                   // a row of taps a block where whole blocks would leave SMs idle
                                                   (p.ca == 64 && ((cin + 31) / 32) * ((cout + 63) / 64) * tiles >= 148
                                                        ? p.rows == 3
                                                        : p.rows == 1));
                ++plans;
                wide += p.ca == 128;
                if (!ok) std::printf("%u %u 2 %u %u %u %d\n", cin, cout, z[1], z[2], z[0], rc);
            }
    std::printf("plans %ld by chunk %ld wide %ld\n", plans, byChunk, wide);
}
