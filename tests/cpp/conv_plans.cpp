// Plans of the 3x3 convolution for every channel count the entry point takes, without a GPU:
// one line "Cin Cout f32 H W B rc" per plan that is refused or that does not hold together.
// Built and run by tests/test_conv_plans.py.
#include <cstdio>

#include "conv_tc.h"

using namespace wrk::conv;

int main() {
    const uint32_t sizes[][3] = {{1, 8, 16}, {1, 64, 128}, {1, 1088, 1920}, {16, 128, 128}};
    long plans = 0, byChunk = 0;
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
                        (p.resident ? !p.byChunk : s.stagesB >= 2);
                    ++plans;
                    byChunk += p.byChunk;
                    if (!ok) std::printf("%u %u %d %u %u %u %d\n", cin, n, f32, z[1], z[2], z[0], rc);
                }
    std::printf("plans %ld by chunk %ld\n", plans, byChunk);
}
