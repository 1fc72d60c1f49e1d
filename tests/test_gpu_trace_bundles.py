"""Batches of more rays than the GPU holds at once: coherent ones (camera rays in pixel order)
and scattered ones run different kernels, which must give what the same rays give in batches
small enough for neither choice.  Bit for bit, at the limit, at one ray more and with a
remainder; and from two threads on one scene."""
import threading

import numpy as np
import pytest

from offlinerenderer_b200 import scenes

pytestmark = pytest.mark.gpu


def _camera_rays(sd, side):
    c = sd.camera
    pos, tgt = np.asarray(c.position, np.float64), np.asarray(c.target, np.float64)
    f = (tgt - pos) / np.linalg.norm(tgt - pos)
    right = np.cross(f, [0.0, 1.0, 0.0])
    right /= np.linalg.norm(right)
    up = np.cross(right, f)
    u = (np.arange(side) + 0.5) / side * 2 - 1
    y, x = np.meshgrid(u, u, indexing="ij")
    d = f + 0.5 * x.reshape(-1, 1) * right + 0.5 * y.reshape(-1, 1) * up
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.empty((side * side, 8), np.float32)
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = pos, 1e-4, d, 1e20
    return r


def _scattered(sd, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = sd.vertices.min(0), sd.vertices.max(0)
    r = np.empty((n, 8), np.float32)
    r[:, 0:3] = lo + (hi - lo) * rng.random((n, 3))
    d = rng.standard_normal((n, 3))
    r[:, 4:7], r[:, 3], r[:, 7] = d / np.linalg.norm(d, axis=1, keepdims=True), 1e-4, 1e20
    return r


def _in_parts(scene, rays):
    t, p, o = [], [], []
    for k in range(0, len(rays), 50000):
        a, b = scene.trace_closest(rays[k:k + 50000])
        t.append(a)
        p.append(b)
        o.append(scene.trace_occluded(rays[k:k + 50000]))
    return np.concatenate(t), np.concatenate(p), np.concatenate(o)


@pytest.mark.parametrize("kind", ["camera", "scattered", "both", "nan"])
@pytest.mark.parametrize("beyond", [0, 1, 12345])
def test_large_batches(gpu, kind, beyond):
    import torch

    sd = scenes.scale_test(8, 8, 1, grid=64, spheres=30)
    scene = gpu.Scene.from_data(sd)
    n = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 128 + beyond
    cam = _camera_rays(sd, int(np.ceil(n ** 0.5)))[:n]
    rays = cam if kind == "camera" else _scattered(sd, n, 3)
    if kind == "both":  # most samples coherent, the rest of the batch not
        rays[: n * 7 // 8] = cam[: n * 7 // 8]
    if kind == "nan":
        rays = cam.copy()
        rays[::7, 4] = np.nan
        rays[5::11, 0] = np.inf
    t, p, o = _in_parts(scene, rays)
    a, b = scene.trace_closest(rays)
    assert np.array_equal(b, p) and np.array_equal(a, t, equal_nan=True)
    assert np.array_equal(scene.trace_occluded(rays), o)


def test_two_threads_on_one_scene(gpu):
    sd = scenes.scale_test(8, 8, 1, grid=64, spheres=30)
    scene = gpu.Scene.from_data(sd)
    batches = [_camera_rays(sd, 600), _scattered(sd, 400000, 5)]
    want = [_in_parts(scene, r) for r in batches]
    bad = []

    def work(k):
        for _ in range(12):
            t, p = scene.trace_closest(batches[k])
            if not (np.array_equal(t, want[k][0]) and np.array_equal(p, want[k][1])):
                bad.append(k)
            if not np.array_equal(scene.trace_occluded(batches[k]), want[k][2]):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k % 2,)) for k in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad


def test_coherent_batches_run_a_thread_per_ray(gpu):
    from torch.profiler import ProfilerActivity, profile
    import torch

    sd = scenes.scale_test(8, 8, 1, grid=64, spheres=30)
    scene = gpu.Scene.from_data(sd)
    times = {}
    for kind, rays in (("camera", _camera_rays(sd, 2048)), ("scattered", _scattered(sd, 1 << 22, 5))):
        scene.trace_closest(rays)
        with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
            scene.trace_closest(rays)
            torch.cuda.synchronize()
        times[kind] = {k: max([e.device_time for e in p.events() if k + "<" in e.name], default=0.0)
                       for k in ("k_query", "k_query_each")}
    if not any(times["camera"].values()):
        pytest.skip("no kernel records on this machine")
    # the kernel that has nothing to do ends at once
    assert times["camera"]["k_query"] < 0.5 * times["camera"]["k_query_each"], times
    assert times["scattered"]["k_query_each"] < 0.5 * times["scattered"]["k_query"], times
