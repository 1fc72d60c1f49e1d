"""The forward convolution at the edges of its plans: output channels split over blocks,
images whose last tile row overhangs, resident and streamed weights, padded and odd
output-channel counts, f32 and bf16 outputs; and the denoiser at sizes where its coarsest
level is one tile.  Against torch in fp32 on the same bf16-rounded operands; the sums run
over 9 * Cin products of unit variance scaled by 1 / sqrt(9 * Cin), so an fp32 sum is
within 1e-5 of the output scale and a bf16 store within half a bf16 ulp (2^-9) more."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _bf(a):
    return torch.tensor(np.asarray(a, np.float32)).to(torch.bfloat16).to(torch.float32)


def _ref(x, w, b, relu):
    y = F.conv2d(_bf(x).permute(0, 3, 1, 2), _bf(w).permute(0, 3, 1, 2), padding=1) + torch.tensor(b).view(1, -1, 1, 1)
    return (F.relu(y) if relu else y).permute(0, 2, 3, 1).numpy()


@pytest.mark.parametrize("cin,cout,h,w", [
    (256, 256, 8, 16),     # one overhanging tile row, channels split over blocks
    (128, 256, 24, 32),    # two tile rows, the second overhanging
    (384, 128, 8, 48),     # the widest input
    (64, 192, 16, 16),     # 192 channels streamed
    (48, 48, 40, 32),      # three 16-channel chunks, resident, 16-channel slices
    (160, 16, 16, 32),     # five 32-channel chunks
    (16, 5, 24, 16),       # padded output channels: element stores
    (64, 64, 328, 640),    # more tiles than the GPU holds at once: every ring wraps
])
@pytest.mark.parametrize("f32", [True, False])
def test_conv_plans(gpu, cin, cout, h, w, f32):
    rng = np.random.default_rng(cin * 7 + cout + h)
    x = rng.standard_normal((1, h, w, cin)).astype(np.float32)
    wt = (rng.standard_normal((cout, 3, 3, cin)) / np.sqrt(9 * cin)).astype(np.float32)
    b = rng.standard_normal(cout).astype(np.float32)
    y = gpu.conv3x3(x, wt, bias=b, relu=True, f32_out=f32)
    ref = _ref(x, wt, b, True)
    tol = 1e-5 * np.abs(ref).max() + (0.0 if f32 else 1.0) * np.abs(ref) * 2.0 ** -8
    assert np.all(np.abs(y - ref) <= tol + 1e-7)


@pytest.mark.parametrize("h,w", [(1, 1), (64, 128), (65, 129), (40, 300)])
def test_denoiser_small_and_odd_frames(gpu, h, w):
    """Cropping and edge clamping: the frame alone and as the corner of its clamped, padded
    self give the same bits."""
    from offlinerenderer_b200 import denoise_train

    rng = np.random.default_rng(h * 1000 + w)
    dn = gpu.Denoiser()
    denoise_train.load_weights(dn)
    img = [rng.random((h, w, 3)).astype(np.float32) for _ in range(3)]
    out = dn.infer(*img)
    hp, wp = (h + 63) // 64 * 64, (w + 127) // 128 * 128
    big = [np.pad(a, ((0, hp - h), (0, wp - w), (0, 0)), mode="edge") for a in img]
    assert np.array_equal(out, dn.infer(*big)[:h, :w])
