"""The forward convolution where an item's input chunks do not fit shared memory together (it
runs chunk by chunk), and where its output channels divide badly.  Against torch in fp64 on
the same bf16-rounded operands.  A sum has 9 * Cin products in steps of 16, each step rounded
or cut to f32 (2^-23 of partial sums that stay below the largest output), so an f32 output is
within 9 * Cin / 16 * 2^-23 of the output scale and a bf16 store within half a bf16 ulp (2^-8
of the value at most) more."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _bf(a):
    return torch.tensor(a).to(torch.bfloat16).to(torch.float64)


@pytest.mark.parametrize("b,cin,cout,h,w", [
    (1, 512, 256, 64, 128),
    (1, 640, 256, 8, 16),     # one tile, channels split over blocks
    (2, 448, 192, 24, 32),    # 192 channels of an item
    (1, 1024, 16, 40, 48),    # the narrowest output
    (1, 528, 64, 24, 16),     # thirty-three 16-channel chunks
    (1, 544, 96, 16, 32),     # 32-channel chunks
    (1, 544, 208, 16, 32),    # 32-channel chunks; 208 channels have no split of at most four
    (1, 176, 208, 24, 32),    # the same where all chunks fit
    (1, 512, 5, 8, 16),       # padded output channels: element stores
    (2, 512, 128, 128, 192),  # more items than blocks: both rings wrap
])
@pytest.mark.parametrize("f32", [True, False])
def test_wide_inputs(gpu, b, cin, cout, h, w, f32):
    rng = np.random.default_rng(cin * 7 + cout + h)
    x = rng.standard_normal((b, h, w, cin)).astype(np.float32)
    wt = (rng.standard_normal((cout, 3, 3, cin)) / np.sqrt(9 * cin)).astype(np.float32)
    bias = rng.standard_normal(cout).astype(np.float32)
    y = gpu.conv3x3(x, wt, bias=bias, relu=True, f32_out=f32)
    ref = F.relu(F.conv2d(_bf(x).cuda().permute(0, 3, 1, 2), _bf(wt).cuda().permute(0, 3, 1, 2),
                          torch.tensor(bias).double().cuda(), padding=1)).permute(0, 2, 3, 1).cpu().numpy()
    tol = 9 * cin / 16 * 2.0 ** -23 * np.abs(ref).max() + (0.0 if f32 else 1.0) * np.abs(ref) * 2.0 ** -8
    assert np.all(np.abs(y - ref) <= tol + 1e-7)
