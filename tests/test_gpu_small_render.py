"""The one-launch renderer of small images against the wavefront kernels (the stage-timed
render always takes those): the same paths, rays and decisions, so the statistics are
equal and a pixel differs by the order of its f32 sums only (the bound the server's
mixed-batch test uses)."""
import dataclasses

import numpy as np
import pytest

from offlinerenderer_b200 import scenes

pytestmark = pytest.mark.gpu

LIMIT = 148 * 4 * 128  # paths the one-launch kernel takes on 148 SMs


def _scene(name):
    if name == "cornell":
        return scenes.cornell(8, 8, 1)
    if name == "showcase":
        return scenes.material_showcase(8, 8, 1, tex_size=64)
    sd = scenes.scale_test(8, 8, 1, grid=64, spheres=40, lights=16)
    rng = np.random.default_rng(3)
    sd.env_map = rng.random((16, 32, 4)).astype(np.float32)
    return sd


def _same(a, b):
    if a is None:
        assert b is None
        return
    nan = np.isnan(b)
    assert np.array_equal(np.isnan(a), nan)
    assert np.all(np.abs(a - b)[~nan] <= 1e-5 * np.abs(b)[~nan] + 1e-6)


@pytest.mark.parametrize("name", ["cornell", "showcase", "terrain"])
@pytest.mark.parametrize("w,h,spp,kw,opts", [
    (64, 64, 1, {}, {}),
    (1, 1, 1, {}, {}),
    (33, 17, 5, dict(useNEE=False), dict(raw_guides=True)),
    (40, 24, 4, dict(maxBounces=1), dict(guides=False)),
    (64, 36, 3, dict(maxBounces=16, fireflyClamp=2.0), dict(max_iterations=20)),
    (57, 31, 2, dict(russianRouletteDepth=0.0), dict(max_iterations=3, sample_offset=9)),
    (48, 48, 2, {}, dict(env_map=True)),
    (296, 256, 1, {}, {}),   # LIMIT paths
    (1943, 39, 1, {}, {}),   # one more: the wavefront both times
])
def test_matches_the_wavefront(gpu, name, w, h, spp, kw, opts):
    sd = _scene(name)
    scene = gpu.Scene.from_data(sd)
    cam = dataclasses.replace(sd.camera, aspect=w / h, lensRadius=0.02 if spp == 3 else 0.0, focalDistance=1.5)
    st = scenes.RenderSettings(w, h, spp, seed=5, **kw)
    r = gpu.Renderer()
    a = r.render(scene, camera=cam, settings=st, **opts)
    b = r.render(scene, camera=cam, settings=st, stage_timing=True, **opts)
    for x, y in ((a.rgb, b.rgb), (a.albedo, b.albedo), (a.normal, b.normal)):
        _same(x, y)
    for k in ("paths", "extensionRays", "shadowRays", "shadowTraced", "bucketPaths", "deviceErrors"):
        assert a.stats[k] == b.stats[k], k
    # whole chunks of 8; the host-driven timed loop sees the end a chunk later
    assert a.stats["iterations"] in (b.stats["iterations"], b.stats["iterations"] - 8) and a.stats["iterations"] % 8 == 0
    assert (w * h * spp <= LIMIT) or w == 1943
