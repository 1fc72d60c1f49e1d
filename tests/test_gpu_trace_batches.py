"""Ray queries at the batch sizes where the persistent query kernel's hand-out of rays can
go wrong (below, at and above a warp, a block and the whole grid), and rays at the edges
of what the node and triangle tests accept.  Exact comparison with the CPU oracle's FP32
intersector, which evaluates the same correctly rounded operations."""
import numpy as np
import pytest

from offlinerenderer_b200 import scenes
from test_gpu_trace import camera_like_rays, random_rays

pytestmark = pytest.mark.gpu

# 148 SMs x 8 blocks x 128 rays: one ray per thread of the whole grid
GRID = 148 * 8 * 128


@pytest.fixture(scope="module")
def showcase(gpu, oracle):
    sd = scenes.material_showcase(64, 64, 1, tex_size=64)
    rays = np.concatenate([camera_like_rays(oracle, sd, GRID // 2 + 64, 3), random_rays(sd, GRID // 2 + 64, 4)])
    rays = rays[np.random.default_rng(5).permutation(len(rays))]
    osc = oracle.scene(sd)
    return gpu.Scene.from_data(sd), rays, osc.closest(rays)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 4097, GRID - 1, GRID, GRID + 1])
def test_batch_sizes(showcase, n):
    scene, rays, (to, po) = showcase
    t, p = scene.trace_closest(rays[:n])
    assert np.array_equal(p, po[:n]) and np.array_equal(t, to[:n])
    occ = scene.trace_occluded(rays[:n])
    assert np.array_equal(occ != 0, po[:n] != 0xFFFFFFFF)


def test_ray_ranges(gpu, oracle):
    """Negative and zero tmin, a tmax in front of, at and behind the hit, NaN rays."""
    sd = scenes.cornell(16, 16, 1)
    scene, osc = gpu.Scene.from_data(sd), oracle.scene(sd)
    rays = random_rays(sd, 4096, 9)
    t, p = scene.trace_closest(rays)
    hit = p != 0xFFFFFFFF
    assert hit.sum() > 1000
    at = rays.copy()
    at[:, 7] = np.where(hit, t, 1e20)  # tmax exactly at the hit: still a hit
    t1, p1 = scene.trace_closest(at)
    assert np.array_equal(t1, t) and np.array_equal(p1, p)
    short = rays[hit].copy()
    short[:, 7] = np.nextafter(t[hit], np.float32(0))
    t2, p2 = scene.trace_closest(short)
    assert not np.any(np.isfinite(t2) & (t2 > short[:, 7]))
    back = rays.copy()
    back[:, 3] = -2.0  # hits behind the origin count too
    to, po = osc.closest(back, mode=1)  # every triangle, FP64
    tb, pb = scene.trace_closest(back)
    # the distance, not the primitive: the boxes' bottom faces lie in the floor's plane
    both = np.isfinite(to) & np.isfinite(tb)
    near = np.abs(tb[both] - to[both]) <= 1e-5 * np.maximum(1.0, np.abs(to[both]))
    assert (np.isfinite(to) == np.isfinite(tb)).mean() >= 0.999 and near.mean() >= 0.999
    assert (tb[both] < 0).any()
    nan = rays[:64].copy()
    nan[:, 4] = np.nan
    tn, pn = scene.trace_closest(nan)
    assert (pn == 0xFFFFFFFF).all() and np.isinf(tn).all()
