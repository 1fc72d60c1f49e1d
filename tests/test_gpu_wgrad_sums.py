"""The weight gradient where a block adds several sums.  All operands are positive, so partial
sums only grow: a step of 16 products cuts at most 2^-22 of the sum so far, n steps at most
n / 2 * 2^-22 of their sum, and adding sums at most 2^-24 of the total each.  The longest sum
has the tiles (of eight steps) that two blocks per SM, of one tap, 128 output and 256 input
channels each, would share.  Against torch in fp64 on the same bf16-rounded operands."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,w,cin,cout", [
    (16, 32, 32, 384, 128),
    (16, 16, 16, 256, 256),
    (4, 64, 64, 256, 256),
    (1, 120, 256, 512, 128),  # the last tile row overhangs
    (2, 64, 96, 240, 64),
    (8, 128, 128, 64, 240),
    (3, 72, 80, 96, 96),
    (1, 256, 256, 256, 16),
    (4, 64, 128, 16, 64),     # 16 input channels, all taps a block
    (1, 24, 48, 16, 64),      # and a row of taps a block
    (1, 128, 128, 512, 512),  # blocks of 128 x 128 channels
    (1, 136, 480, 224, 368),  # their last channels past the end, and an overhanging tile row
    (1, 200, 320, 128, 128),
])
def test_several_sums(gpu, b, h, w, cin, cout):
    rng = np.random.default_rng(cin * 5 + cout + h)
    x = rng.random((b, h, w, cin)).astype(np.float32)
    g = rng.random((b, h, w, cout)).astype(np.float32)
    _check(gpu.conv3x3_wgrad(g, x), x, g)


def _check(dw, x, g):
    (b, h, w, cin), cout = x.shape, g.shape[3]
    bf = lambda a: torch.tensor(a, device="cuda").to(torch.bfloat16).to(torch.float64)
    xp, gf = torch.nn.functional.pad(bf(x), (0, 0, 1, 1, 1, 1)), bf(g).reshape(-1, cout)
    ref = torch.stack([torch.stack([gf.T @ xp[:, dy:dy + h, dx:dx + w].reshape(-1, cin) for dx in range(3)], 1)
                       for dy in range(3)], 1).cpu().numpy()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = b * (w // 8) * -(-h // 16)
    cells = 9 * -(-cin // 256) * -(-cout // 128)
    parts = min(-(-2 * sms // cells), tiles)
    longest = -(-tiles // parts)
    tol = 8 * longest / 2 * 2.0 ** -22 + -(-tiles // longest) * 2 * 2.0 ** -24
    assert np.all(np.abs(dw - ref) <= tol * ref)


def test_gradient_at_any_float_address(gpu):
    """The 16-byte atomics are for gradients at a multiple of 16 bytes; others take 4-byte ones."""
    rng = np.random.default_rng(2)
    b, h, w, cin, cout = 1, 16, 32, 48, 80
    x = rng.random((b, h, w, cin)).astype(np.float32)
    g = rng.random((b, h, w, cout)).astype(np.float32)
    dx, dg = (torch.tensor(a, device="cuda").to(torch.bfloat16) for a in (x, g))
    buf = torch.zeros(cout * 9 * cin + 2, device="cuda")
    torch.cuda.synchronize()
    assert gpu.lib().wrk_conv3x3_wgrad(dg.data_ptr(), dx.data_ptr(), b, h, w, cin, cout, buf.data_ptr() + 4) == 0
    out = buf.cpu().numpy()
    assert out[0] == 0.0 and out[-1] == 0.0
    _check(out[1:-1].reshape(cout, 3, 3, cin), x, g)
