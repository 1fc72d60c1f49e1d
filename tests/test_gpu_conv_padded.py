"""The forward convolution with output channels that are no multiple of 16: rows of whole
16-byte units leave by TMA without the padding channels, others by plain stores, and so do
outputs at addresses TMA cannot take.  Against torch in fp64 on the same bf16-rounded operands;
tolerances as in test_gpu_conv_wide.py.  Nothing past an output is touched."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _run(gpu, x, wt, bias, out, f32):
    b, h, w, cin = x.shape
    rc = gpu.lib().wrk_conv3x3_forward(x.data_ptr(), b, h, w, cin, wt.data_ptr(), bias.data_ptr(), wt.shape[0], 2 * f32,
                                       out.data_ptr())
    assert rc == 0, gpu.lib().wrk_last_error().decode()


@pytest.mark.parametrize("cin,cout,h,w", [
    (64, 3, 24, 16), (64, 8, 24, 32), (16, 24, 40, 16), (64, 72, 16, 48), (96, 100, 24, 16), (64, 136, 8, 32),
    (256, 200, 16, 16), (64, 250, 16, 32), (512, 72, 8, 16), (128, 249, 8, 16),
])
@pytest.mark.parametrize("f32", [1, 0])
@pytest.mark.parametrize("shift", [0, 1])  # elements past a 256-byte boundary
def test_padded_channels(gpu, cin, cout, h, w, f32, shift):
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn((2, h, w, cin), device="cuda", generator=g).bfloat16()
    wt = (torch.randn((cout, 3, 3, cin), device="cuda", generator=g) / (9 * cin) ** 0.5).bfloat16()
    bias = torch.randn(cout, device="cuda", generator=g)
    n = 2 * h * w * cout
    buf = torch.full((n + shift + 64,), 7.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    torch.cuda.synchronize()
    _run(gpu, x, wt, bias, buf[shift:], f32)
    assert (buf[:shift] == 7.0).all() and (buf[shift + n:] == 7.0).all()
    y = buf[shift:shift + n].double().reshape(2, h, w, cout)
    ref = F.conv2d(x.double().permute(0, 3, 1, 2), wt.double().permute(0, 3, 1, 2), bias.double(), padding=1).permute(0, 2, 3, 1)
    tol = 9 * cin / 16 * 2.0 ** -23 * ref.abs().max() + (0.0 if f32 else 1.0) * ref.abs() * 2.0 ** -8
    assert ((y - ref).abs() <= tol + 1e-7).all()


@pytest.mark.parametrize("cout", [72, 200])
@pytest.mark.parametrize("f32", [1, 0])
def test_padded_channels_cost_what_whole_ones_cost(gpu, cout, f32):
    """The same work items as the next multiple of 16: at most twice its device time (as plain
    stores they took five to seven times)."""
    from torch.profiler import ProfilerActivity, profile

    times = []
    for n in (cout, cout + 8):
        x = torch.randn((1, 512, 512, 64), device="cuda").bfloat16()
        wt = torch.randn((n, 3, 3, 64), device="cuda").bfloat16()
        bias, y = torch.randn(n, device="cuda"), torch.empty((1, 512, 512, n), device="cuda",
                                                               dtype=torch.float32 if f32 else torch.bfloat16)
        torch.cuda.synchronize()
        _run(gpu, x, wt, bias, y, f32)
        with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
            for _ in range(5):
                _run(gpu, x, wt, bias, y, f32)
            torch.cuda.synchronize()
        t = sorted(e.device_time for e in p.events() if "k_conv_fwd" in e.name)
        if not t:
            pytest.skip("no kernel records on this machine")
        times.append(t[len(t) // 2])
    assert times[0] <= 2.0 * times[1], times
