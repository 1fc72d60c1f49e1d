"""A render that fails on the device leaves the caller's images as they were, whichever
kernels ran it.  The scene: a million copies of one right triangle, and rays through the
other half of their boxes, so a ray misses every triangle but has to visit every node; it
gives up at 65,536 and sets the error flag."""
import numpy as np
import pytest

from offlinerenderer_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage_timing", [False, True])
def test_images_are_untouched(gpu, stage_timing):
    import torch

    b = scenes._Builder()
    b.mesh([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.tile(np.arange(3, dtype=np.uint32), 1 << 20), b.lambertian((0.5, 0.5, 0.5)))
    cam = scenes.Camera(position=(0.9, 0.9, -5.0), target=(0.9, 0.9, 0.0), fovY=0.01, aspect=1.0)
    sd = b.build(env=(1, 1, 1), camera=cam, settings=scenes.RenderSettings(4, 4, 1))
    scene, r = gpu.Scene.from_data(sd), gpu.Renderer()
    out = tuple(np.full((4, 4, 3), 7.0, np.float32) for _ in range(3))
    with pytest.raises(gpu.WrkError, match="device error flags"):
        r.render(scene, out=out, stage_timing=stage_timing)
    assert all((a == 7.0).all() for a in out)
    dev = [torch.full((4, 4, 3), 7.0, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    with pytest.raises(gpu.WrkError, match="device error flags"):
        r.render_device(scene, *(gpu.TensorPtr(t) for t in dev[:1]), d_albedo=gpu.TensorPtr(dev[1]),
                        d_normal=gpu.TensorPtr(dev[2]), stage_timing=stage_timing)
    assert all((t == 7.0).all().item() for t in dev)
    # and the renderer goes on
    ok = scenes.cornell(16, 16, 4)
    ref = gpu.Renderer().render(gpu.Scene.from_data(ok))
    assert np.allclose(r.render(gpu.Scene.from_data(ok)).rgb, ref.rgb, rtol=1e-5, atol=1e-6)
