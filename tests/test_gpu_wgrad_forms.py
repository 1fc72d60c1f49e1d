"""The weight gradient at the edges of its plans: one to many blocks of 16, 32 and 64 output
and of 16 and 32 input channels, tiles that overhang the image, fewer tiles than SMs and more.
Against torch in fp64 on the same bf16-rounded operands: the products are exact in fp32, and
a block adds at most 512 sums of 16 of them to partial sums no larger than twice the largest
gradient, so the error is within 512 * 2 * 2^-23 < 1.3e-4 of it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,w,cin,cout", [
    (1, 8, 16, 16, 16),     # half a tile high
    (1, 24, 48, 32, 16),    # the second tile row overhangs
    (2, 40, 16, 48, 32),    # three blocks of 16 channels
    (1, 16, 16, 96, 32),    # three blocks of 32, two tiles
    (3, 8, 32, 384, 64),    # twelve blocks of input channels
    (2, 64, 64, 64, 64),
    (2, 24, 48, 16, 64),
    (4, 128, 160, 32, 32),  # more tiles than SMs
    (1, 16, 32, 32, 48),    # three blocks of 16 output channels
    (1, 24, 32, 64, 128),
    (2, 16, 16, 256, 256),  # more cells than two blocks per SM leave splits for
    (1, 16, 16, 512, 144),  # the widest input
])
def test_wgrad_plans(gpu, b, h, w, cin, cout):
    rng = np.random.default_rng(cin * 5 + cout + h)
    bf = lambda a: torch.tensor(a).to(torch.bfloat16).to(torch.float64)
    x = rng.standard_normal((b, h, w, cin)).astype(np.float32)
    g = rng.standard_normal((b, h, w, cout)).astype(np.float32)
    dw = gpu.conv3x3_wgrad(g, x)
    ref = torch.nn.grad.conv2d_weight(bf(x).permute(0, 3, 1, 2), (cout, cin, 3, 3), bf(g).permute(0, 3, 1, 2),
                                      padding=1).permute(0, 2, 3, 1).numpy()
    assert np.abs(dw - ref).max() <= 1.3e-4 * np.abs(ref).max()
