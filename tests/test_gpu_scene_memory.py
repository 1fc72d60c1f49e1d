"""Device memory of a resident scene: its arrays, 48 bytes of triangle record and 80 of pair
record a triangle, and 80 a possible 8-wide node, of which there are at most as many as inner
nodes in a binary tree with one triangle a leaf (one less than triangles)."""
import numpy as np
import pytest

from offlinerenderer_b200 import scenes

pytestmark = pytest.mark.gpu


def test_resident_bytes_per_triangle(gpu):
    import torch

    n = 1 << 20
    rng = np.random.default_rng(1)
    b = scenes._Builder()
    v = (rng.random((n, 1, 3)) + 0.01 * rng.random((n, 3, 3))).astype(np.float32)
    b.mesh(v, np.arange(3 * n, dtype=np.uint32), b.lambertian((0.5, 0.5, 0.5)))
    cam = scenes.Camera(position=(0.5, 0.5, -3.0), target=(0.5, 0.5, 0.5), fovY=0.6, aspect=1.0)
    sd = b.build(env=(1, 1, 1), camera=cam, settings=scenes.RenderSettings(8, 8, 1))
    first = gpu.Scene.from_data(sd)  # the build's scratch pool keeps its memory
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    scene = gpu.Scene.from_data(sd)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    arrays = sd.vertices.nbytes + 12 * n + 4 * n + (0 if sd.normals is None else sd.normals.nbytes) + \
        (0 if sd.uvs is None else sd.uvs.nbytes)
    assert used <= arrays + (48 + 80 + 80) * n + (8 << 20), used / n
    del first, scene
