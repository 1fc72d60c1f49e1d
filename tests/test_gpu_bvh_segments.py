"""BVH builds whose levels put many tasks into one block of the builder's kernels: clusters
just above the small-task size, coincident clusters (object-median splits), and primitive
counts at the edges of a block.  The tree is validated on the CPU and traced there with
the same correctly rounded tests, so the comparison is exact."""
import numpy as np
import pytest

from offlinerenderer_b200 import scenes
from test_gpu_trace import random_rays

pytestmark = pytest.mark.gpu


def clustered(n, per, coincident, seed):
    rng = np.random.default_rng(seed)
    k = np.arange(n) // per
    centre = rng.uniform(-10, 10, (k[-1] + 1, 3))[k]
    if coincident:
        tri = centre[:, None] + rng.uniform(-0.3, 0.3, (k[-1] + 1, 3, 3))[k]
    else:
        tri = centre[:, None] + rng.uniform(-0.3, 0.3, (n, 3, 3))
    mats = scenes.cornell(8, 8, 1).materials[:1]
    return scenes.SceneData(vertices=tri.reshape(-1, 3).astype(np.float32),
                            indices=np.arange(3 * n, dtype=np.uint32).reshape(n, 3),
                            tri_material=np.zeros(n, np.uint32), materials=mats)


@pytest.mark.parametrize("n,per,coincident", [
    (1, 1, False), (2, 1, False), (16, 16, False), (17, 17, True), (255, 17, False), (256, 17, True), (257, 18, False),
    (1000, 200, True), (5000, 17, False), (5000, 19, True), (20000, 40, False)])
def test_clusters(gpu, oracle, n, per, coincident):
    sd = clustered(n, per, coincident, n)
    s = gpu.Scene.from_data(sd)
    nodes, tris = s.bvh_export()
    rc, depth, internal, leaf = oracle.bvh8_validate(nodes, tris)
    assert rc == 0 and depth == s.bvh_info()["depth"] and internal == nodes.shape[0] - 1
    rays = random_rays(sd, 4096, 2)
    t, p, _, _ = oracle.bvh8_trace(nodes, tris, rays)
    tg, pg = s.trace_closest(rays)
    # (coincident triangles tie: the distance is the result there, not which of them it was)
    assert np.array_equal(t, tg) and (coincident or np.array_equal(p, pg))
