"""Which kernels a render runs, from the device's own launch records (CUPTI, through torch's
profiler): one launch where every path has a resident thread and a place in the queues, the
wavefront above either limit and when its stages are timed.  test_gpu_small_render.py compares
the two routes' results; this shows that they are two."""
import pytest

from offlinerenderer_b200 import scenes

pytestmark = pytest.mark.gpu


def _kernels(f):
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
        f()
    return " ".join(e.name for e in p.events() if "wrk::k_" in e.name)


def test_one_launch_up_to_its_limits(gpu):
    import torch

    scene = gpu.Scene.from_data(scenes.cornell(8, 8, 1))
    limit = torch.cuda.get_device_properties(0).multi_processor_count * 4 * 128  # resident threads
    small = 1 << 14  # paths a renderer with that queue capacity takes at once
    torch.cuda.synchronize()
    # (capacity, width, height, stage timing, one launch)
    cases = [(0, limit // 128, 128, False, True), (0, limit // 128 + 1, 128, False, False), (0, 64, 64, True, False),
             (small, 128, 128, False, True), (small, 129, 128, False, False)]
    for capacity, w, h, timing, one in cases:
        r = gpu.Renderer(capacity=capacity)
        render = lambda: r.render(scene, settings=scenes.RenderSettings(w, h, 1), stage_timing=timing)
        render()
        names = _kernels(render)
        if not names:
            pytest.skip("no kernel records on this machine")
        assert ("k_render_small" in names) == one, (capacity, w, h, names)
        assert ("k_trace_persistent" in names) != one, (capacity, w, h, names)
