"""The work a user of this framework has it do, as measurable cases.

A case is a dict of plain values; ``prepare(case, seed)`` makes what a program holds
before the call (scene, renderer, server, denoiser, images on the GPU), ``run(state)``
is one pass through the public entry points, and ``work(case)`` is what that pass cannot
do without.  ``listed()`` are fixed cases over the framework's range, ``draw(rng)`` gives
others of the same ranges.

Kinds (``case["kind"]``):
  render    ``Renderer.render`` / ``render_device`` of a resident scene
  serve     a batch of requests through one ``Server``
  finalize  a new scene: upload, light CDF, BVH build, first ray queries
  rays      closest-hit and occlusion queries of a batch of rays in device memory
  denoise   ``Denoiser.infer_device``
  train     forward + backward pass of the denoiser (loss and gradients)
  tonemap   the 8-bit output image of a rendered frame
"""
from __future__ import annotations

import dataclasses
import math
import os

import numpy as np
import torch
import torch.nn.functional as F

from offlinerenderer_b200 import denoise_train, scenes, wrk


def _render(name, scene, width, height, spp, **kw):
    case = dict(kind="render", scene=scene, width=width, height=height, spp=spp, bounces=8, nee=True, guides=True,
                env_map=False, lens=0.0, clamp=0.0, capacity=0, host=True)
    case.update(kw)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # An interactive preview while a camera is being placed: the smallest call, host image out.
        _render("preview_64", "cornell", 64, 64, 1),
        # The plain Cornell configuration (256 x 256, 64 spp), image and guides to the host.
        _render("cornell_256_64spp", "cornell", 256, 256, 64),
        # The material showcase the benchmark times (512 x 512, 256 spp, depth 16), into device
        # memory, with queues of the size the autotuner chooses for a workload of this size.
        _render("showcase_512_256spp", "showcase", 512, 512, 256, bounces=16, capacity=1 << 25, host=False),
        # The scale scene (2.4M triangles) as a low-sample full-HD frame, ready for the denoiser.
        _render("terrain_1080p_4spp", "terrain1024", 1920, 1080, 4, host=False),
        # An odd-sized frame with the less common options: environment map, thin lens,
        # firefly clamp, no guides, and an odd sample count.
        _render("odd_333x217_7spp", "showcase", 333, 217, 7, bounces=5, guides=False, env_map=True, lens=0.02,
                clamp=10.0),
        # A few mixed requests arriving together at a server with two resident scenes, denoised.
        dict(name="serve_6_requests", kind="serve", requests=6, largest=512, spp=4, denoise=True),
        # A program that loads a new scene: upload, lights, BVH, and its first ray queries.
        dict(name="finalize_676k_tris", kind="finalize", grid=512, spheres=120, rays=65536),
        # Picking / visibility queries of a batch of rays (half from the camera, half scattered).
        dict(name="rays_1m", kind="rays", scene="terrain512", rays=1 << 20),
        # Denoising a full-HD frame; an odd-sized small one, as a preview does after every pass.
        dict(name="denoise_1080p", kind="denoise", batch=1, width=1920, height=1080),
        dict(name="denoise_300x170", kind="denoise", batch=1, width=300, height=170),
        # One forward + backward pass of denoiser training at the trainer's batch of crops.
        dict(name="train_16x128", kind="train", batch=16, width=128, height=128),
        # The 8-bit image of a 4K frame, as every program that saves a PNG makes it.
        dict(name="tonemap_4k", kind="tonemap", width=3840, height=2160),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["render"] * 6 + ["serve", "finalize", "rays", "denoise", "denoise", "train", "tonemap"])
    if kind == "render":
        scene = rng.choice(["cornell", "showcase", "variant", "terrain512", "terrain1024"])
        w, h = _log_int(rng, 40, 1920), _log_int(rng, 40, 1080)
        if rng.random() < 0.5:  # multiples of 8 are as common as odd sizes
            w, h = (w + 7) // 8 * 8, (h + 7) // 8 * 8
        # samples in all: no more than half of the showcase's, and of the scale scene a fraction
        most = (1 << 25) if not scene.startswith("terrain") else 1 << 23
        spp = _log_int(rng, 1, max(1, min(256, most // (w * h))))
        return _render(None, scene, w, h, spp, bounces=rng.choice([1, 4, 8, 8, 16]), nee=rng.random() < 0.85,
                       guides=rng.random() < 0.7, env_map=rng.random() < 0.2, lens=rng.choice([0.0, 0.0, 0.0, 0.02]),
                       clamp=rng.choice([0.0, 0.0, 10.0]), capacity=rng.choice([0, 0, 1 << 18, 1 << 20, 1 << 24]),
                       host=rng.random() < 0.5)
    if kind == "serve":
        return dict(kind="serve", requests=rng.randint(1, 12), largest=_log_int(rng, 64, 512), spp=rng.choice([1, 2, 4, 8]),
                    denoise=rng.random() < 0.6)
    if kind == "finalize":
        return dict(kind="finalize", grid=_log_int(rng, 16, 512), spheres=rng.randint(1, 120),
                    rays=_log_int(rng, 1024, 65536))
    if kind == "rays":
        return dict(kind="rays", scene=rng.choice(["cornell", "showcase", "variant", "terrain512"]),
                    rays=_log_int(rng, 1000, 1 << 22))
    if kind == "denoise":
        b = rng.choice([1, 1, 1, 2, 4])
        return dict(kind="denoise", batch=b, width=_log_int(rng, 40, 1920), height=_log_int(rng, 40, 1080 // b))
    if kind == "train":
        return dict(kind="train", batch=rng.randint(1, 16), width=128 * rng.randint(1, 2), height=64 * rng.randint(1, 2))
    return dict(kind="tonemap", width=_log_int(rng, 60, 3840), height=_log_int(rng, 60, 2160))


# ---- inputs ---------------------------------------------------------------------------
def _scene_data(name, seed, width=64, height=64):
    if name == "cornell":
        return scenes.cornell(width, height, 1, seed=seed + 1)
    if name == "showcase":
        return scenes.material_showcase(width, height, 1, seed=seed + 1)
    if name == "variant":
        return scenes.cornell_variant(seed)
    grid = int(name[len("terrain"):])
    return scenes.scale_test(width, height, 1, seed=seed + 1, grid=grid, spheres=250 if grid >= 1024 else 120)


def _sky(seed):
    """A small lat-long map: a horizon gradient and a sun."""
    rng = np.random.default_rng(seed)
    v, u = np.mgrid[0:64, 0:128]
    m = np.zeros((64, 128, 4), np.float32)
    m[..., :3] = (0.2 + 0.8 * v[..., None] / 64.0) * rng.uniform(0.3, 1.0, 3)
    d = np.hypot((u - rng.uniform(20, 100)) / 4.0, (v - 12) / 4.0)
    m[..., :3] += (30.0 * np.exp(-d * d))[..., None]
    return m


def _images(batch, height, width, seed):
    """A noisy HDR frame with its first-hit guides: smooth structure, albedo edges, unit
    normals, and log-normal noise with fireflies on the radiance."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def smooth(c, cells):
        x = torch.rand((batch, c, max(2, height // cells), max(2, width // cells)), device="cuda", generator=g)
        return F.interpolate(x, size=(height, width), mode="bilinear", align_corners=False).permute(0, 2, 3, 1).contiguous()

    alb = (smooth(3, 48) > 0.5).float() * 0.6 + 0.2 * smooth(3, 12)
    nrm = F.normalize(smooth(3, 32) * 2.0 - 1.0, dim=-1)
    clean = alb * smooth(3, 64) * 2.0
    noise = torch.exp(0.6 * torch.randn(clean.shape, device="cuda", generator=g))
    rgb = clean * noise
    rgb = torch.where(torch.rand(clean.shape[:3] + (1,), device="cuda", generator=g) < 1e-3, rgb * 40.0, rgb)
    return rgb.contiguous(), alb.contiguous(), nrm.contiguous(), clean.contiguous()


def _camera(sd, seed, width, height, lens):
    """The scene's camera, moved a little as a user's would be."""
    rng = np.random.default_rng(seed)
    c = sd.camera
    pos = tuple(float(p + d) for p, d in zip(c.position, rng.uniform(-0.03, 0.03, 3)))
    return dataclasses.replace(c, position=pos, aspect=float(np.float32(width) / np.float32(height)), lensRadius=lens,
                               focalDistance=1.9 if lens > 0.0 else 0.0)


def _rays(sd, n, seed):
    """Half the rays from the scene's camera, half from scattered points in its bounds."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo = torch.tensor(sd.vertices.min(0), device="cuda")
    hi = torch.tensor(sd.vertices.max(0), device="cuda")
    k = n // 2
    tgt = lo + (hi - lo) * torch.rand((n, 3), device="cuda", generator=g)
    org = lo + (hi - lo) * torch.rand((n, 3), device="cuda", generator=g)
    org[:k] = torch.tensor(sd.camera.position, device="cuda", dtype=torch.float32)
    d = F.normalize(tgt - org + 1e-4, dim=-1)
    rays = torch.empty((n, 8), device="cuda")
    rays[:, 0:3], rays[:, 3], rays[:, 4:7], rays[:, 7] = org, 1e-4, d, 1e20
    return rays


def _denoiser(seed):
    dn = wrk.Denoiser(seed=seed % 1000 + 1)
    denoise_train.load_weights(dn)
    return dn


def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind == "render":
        w, h = case["width"], case["height"]
        sd = _scene_data(case["scene"], seed % 10000, w, h)
        sd.env_map = _sky(seed) if case["env_map"] else None
        s["scene"] = wrk.Scene.from_data(sd)
        s["renderer"] = wrk.Renderer(capacity=case["capacity"])
        s["camera"] = _camera(sd, seed, w, h, case["lens"])
        s["settings"] = scenes.RenderSettings(w, h, case["spp"], maxBounces=case["bounces"], useNEE=case["nee"],
                                              fireflyClamp=case["clamp"], seed=seed % 100000 + 1)
        n = 3 if case["guides"] else 1
        if case["host"]:
            pinned = [torch.empty((h, w, 3), pin_memory=True).numpy() for _ in range(n)]
            s["out"] = tuple(pinned + [None] * (3 - n))
        else:
            s["out"] = [torch.empty((h, w, 3), device="cuda") for _ in range(n)]
    elif kind == "serve":
        rng = np.random.default_rng(seed)
        sds = [_scene_data("terrain256", seed % 10000), _scene_data("showcase", seed % 10000)]
        s["scenes"] = [wrk.Scene.from_data(sd) for sd in sds]
        s["server"] = wrk.Server()
        s["denoiser"] = _denoiser(seed)
        s["server"].set_denoiser(s["denoiser"])
        s["requests"] = []
        for k in range(case["requests"]):
            side = case["largest"] >> (k % 3)
            w, h = max(16, side + (k % 2) * 5), max(16, side * 3 // 4)
            cam = _camera(sds[k % 2], int(rng.integers(1 << 30)), w, h, 0.0)
            st = scenes.RenderSettings(w, h, case["spp"], seed=int(rng.integers(1, 1 << 30)))
            s["requests"].append((s["scenes"][k % 2], cam, st))
    elif kind == "finalize":
        s["data"] = scenes.scale_test(64, 64, 1, seed=seed % 10000 + 1, grid=case["grid"], spheres=case["spheres"])
        s["rays"] = _rays(s["data"], case["rays"], seed).cpu().numpy()
    elif kind == "rays":
        sd = _scene_data(case["scene"], seed % 10000)
        s["scene"] = wrk.Scene.from_data(sd)
        s["rays"] = _rays(sd, case["rays"], seed)
        n = case["rays"]
        s["t"] = torch.empty(n, device="cuda")
        s["prim"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["occluded"] = torch.empty(n, dtype=torch.int32, device="cuda")
    elif kind in ("denoise", "train"):
        s["images"] = _images(case["batch"], case["height"], case["width"], seed)
        s["denoiser"] = _denoiser(seed)
        s["out"] = torch.empty_like(s["images"][0])
        if kind == "train":
            s["grads"] = torch.empty(s["denoiser"].num_params, device="cuda")
    else:
        s["rgb"] = _images(1, case["height"], case["width"], seed)[0]
        s["bytes"] = torch.empty(s["rgb"].shape, dtype=torch.uint8, device="cuda")
    return s


# ---- one pass -------------------------------------------------------------------------
def _ok(rc):
    if rc:
        raise wrk.WrkError(rc, wrk.lib().wrk_last_error().decode())


def _run_render(s):
    case = s["case"]
    if case["host"]:
        r = s["renderer"].render(s["scene"], camera=s["camera"], settings=s["settings"], guides=case["guides"],
                                 env_map=case["env_map"], out=s["out"])
        out = {"rgb": r.rgb, "albedo": r.albedo, "normal": r.normal}
        stats = r.stats
    else:
        t = [wrk.TensorPtr(x) for x in s["out"]]
        if case["env_map"]:  # render_device has no such option: the C entry point takes it as a flag
            p = wrk.params_struct(s["settings"], env_map=True)
            cam, st = wrk.camera_struct(s["camera"]), wrk.RenderStatsC()
            _ok(wrk.lib().wrk_render_device(s["renderer"].handle, s["scene"].handle, cam, p, t[0].ptr,
                                            t[1].ptr if case["guides"] else None, t[2].ptr if case["guides"] else None, st))
            stats = {"paths": st.paths, "extensionRays": st.extensionRays, "shadowRays": st.shadowRays}
        else:
            stats = s["renderer"].render_device(s["scene"], t[0], camera=s["camera"], settings=s["settings"],
                                                d_albedo=t[1] if case["guides"] else None,
                                                d_normal=t[2] if case["guides"] else None)
        out = dict(zip(("rgb", "albedo", "normal"), s["out"]))
    for k in ("paths", "extensionRays", "shadowRays"):
        out[k] = int(stats[k])
    return out


def _run_serve(s):
    srv = s["server"]
    tickets = [srv.submit(sc, camera=cam, settings=st, denoise=s["case"]["denoise"]) for sc, cam, st in s["requests"]]
    out = []
    for t in tickets:
        srv.wait(t)
        out.append(srv.result(t)[:3])
    return out


def _run_finalize(s):
    scene = wrk.Scene.from_data(s["data"])
    t, prim = scene.trace_closest(s["rays"])
    tris, cdf = scene.light_cdf()
    return {"t": t, "prim": prim, "light_triangles": tris, "light_cdf": cdf}


def _run_rays(s):
    n, L, h, r = s["case"]["rays"], wrk.lib(), s["scene"].handle, wrk.TensorPtr(s["rays"])
    _ok(L.wrk_trace_closest(h, r.ptr, n, s["t"].data_ptr(), s["prim"].data_ptr()))
    _ok(L.wrk_trace_occluded(h, r.ptr, n, s["occluded"].data_ptr()))
    return {"t": s["t"], "prim": s["prim"], "occluded": s["occluded"]}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "render":
        return _run_render(s)
    if kind == "serve":
        return _run_serve(s)
    if kind == "finalize":
        return _run_finalize(s)
    if kind == "rays":
        return _run_rays(s)
    if kind == "tonemap":
        _ok(wrk.lib().wrk_tonemap_aces(wrk.TensorPtr(s["rgb"]).ptr, case["width"] * case["height"], s["bytes"].data_ptr()))
        return s["bytes"]
    rgb, alb, nrm, target = (wrk.TensorPtr(x) for x in s["images"])
    b, h, w = case["batch"], case["height"], case["width"]
    if kind == "denoise":
        s["denoiser"].infer_device(rgb, alb, nrm, b, h, w, wrk.TensorPtr(s["out"]))
        return s["out"]
    loss = s["denoiser"].gradients_device(rgb, alb, nrm, target, b, h, w)
    s["denoiser"].grads_copy(s["grads"].data_ptr())
    return {"loss": loss, "grads": s["grads"]}


# ---- what a pass cannot do without ------------------------------------------------------
# 3x3 convolutions of the denoiser: (Cin, Cout, level); the head stores 3 of its channels.
LAYERS = [(16, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 128, 2), (128, 128, 2), (128, 256, 3), (256, 256, 3),
          (384, 128, 2), (128, 128, 2), (192, 64, 1), (64, 64, 1), (96, 32, 0), (32, 32, 0), (32, 3, 0)]
UNET_PARAMS = sum(co * (9 * ci + 1) for ci, co, _ in LAYERS)
# A path of these scenes takes about four closest-hit rays and three shadow queries; a ray
# about four 8-wide node tests (8 boxes x 12 operations) and four triangle tests (30), a
# hit about 200 operations of shading.
RAYS_PER_PATH, FLOPS_PER_RAY, FLOPS_PER_HIT = 7, 4 * (8 * 12 + 30), 200
TRIANGLES = {"cornell": 36, "showcase": 15372, "variant": 20000, "terrain256": 284000, "terrain512": 675906,
             "terrain1024": 2413122}


def _trace_work(rays, triangles):
    # the part of the tree that the rays can touch: at most all of it (about 100 bytes a triangle)
    return min(100 * triangles, 500 * rays), rays * FLOPS_PER_RAY


def work(case):
    kind = case["kind"]
    if kind == "render":
        px = case["width"] * case["height"]
        paths = px * case["spp"]
        per_path = RAYS_PER_PATH if case["nee"] else 4
        b, f = _trace_work(paths * per_path, TRIANGLES[case["scene"]])
        return {"bytes": b + px * 12 * (3 if case["guides"] else 1), "flops": f + paths * 4 * FLOPS_PER_HIT}
    if kind == "serve":
        b = f = 0
        for k in range(case["requests"]):
            side = case["largest"] >> (k % 3)
            px = max(16, side + (k % 2) * 5) * max(16, side * 3 // 4)
            tb, tf = _trace_work(px * case["spp"] * RAYS_PER_PATH, TRIANGLES["showcase" if k % 2 else "terrain256"])
            b += tb + px * 36
            f += tf + px * case["spp"] * 4 * FLOPS_PER_HIT
            if case["denoise"]:
                f += sum(18 * ci * co * px / 4 ** lv for ci, co, lv in LAYERS)
        return {"bytes": b, "flops": f}
    if kind == "finalize":
        tris = 2 * (case["grid"] - 1) ** 2 + 1280 * case["spheres"] + 64
        verts = case["grid"] ** 2 + 642 * case["spheres"] + 192
        # scene in (vertices, normals, uvs where it has them, indices, materials), tree out; a binned build
        # touches every triangle's box once per binary level
        levels = math.log2(tris)
        return {"bytes": verts * 24 + tris * 16 + tris * 100 + case["rays"] * 40, "flops": tris * levels * 30}
    if kind == "rays":
        b, f = _trace_work(2 * case["rays"], TRIANGLES[case["scene"]])
        return {"bytes": b + case["rays"] * (32 + 12), "flops": f}
    px = case.get("batch", 1) * case["width"] * case["height"]
    if kind == "tonemap":
        return {"bytes": px * 15, "flops": px * 3 * 40}
    conv = sum(18 * ci * co * px / 4 ** lv for ci, co, lv in LAYERS)
    if kind == "denoise":
        return {"bytes": px * 48 + UNET_PARAMS * 2, "flops": conv}
    # backward: weight gradients of every layer, data gradients of all but the first
    return {"bytes": px * 48 + UNET_PARAMS * 6, "flops": 3 * conv - 18 * 16 * 32 * px}


# ---- 64-bit values ----------------------------------------------------------------------
def _weights64():
    path = os.path.join(os.path.dirname(denoise_train.__file__), "weights", "unet_scale.wrkw")
    with open(path, "rb") as f:
        if f.read(8) != b"WRKUNET1":
            raise ValueError(path)
        count, _ = np.frombuffer(f.read(16), "<u8")
        bits = np.frombuffer(f.read(2 * int(count)), "<u2").astype(np.uint32) << 16
    flat = torch.from_numpy(bits.view(np.float32).astype(np.float64)).cuda()
    out, o = [], 0
    for ci, co, _ in LAYERS:
        w = flat[o:o + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous()
        b = flat[o + co * 9 * ci:o + co * (9 * ci + 1)].clone()
        o += co * (9 * ci + 1)
        out.append((w, b))
    return out


def _unet64(rgb, alb, nrm, params):
    """The network in 64 bits on [B, H, W, 3] images (H a multiple of 64, W of 128): the
    prediction log1p(radiance) + residual."""
    lg = torch.log1p(rgb.double().clamp_min(0.0))
    x = torch.cat([lg, alb.double(), nrm.double(), torch.zeros_like(lg), torch.zeros_like(lg), lg[..., :1] * 0.0], -1)
    x = x.permute(0, 3, 1, 2)

    def conv(i, v, relu=True):
        v = F.conv2d(v, params[i][0], params[i][1], padding=1)
        return F.relu(v) if relu else v

    def up(v):
        return F.interpolate(v, scale_factor=2, mode="nearest")

    s0 = conv(1, conv(0, x))
    s1 = conv(3, conv(2, F.avg_pool2d(s0, 2)))
    s2 = conv(5, conv(4, F.avg_pool2d(s1, 2)))
    d = conv(7, conv(6, F.avg_pool2d(s2, 2)))
    d = conv(9, conv(8, torch.cat([up(d), s2], 1)))
    d = conv(11, conv(10, torch.cat([up(d), s1], 1)))
    d = conv(13, conv(12, torch.cat([up(d), s0], 1)))
    return lg + conv(14, d, relu=False).permute(0, 2, 3, 1)


def exact(case, seed):
    if case["kind"] == "denoise":
        rgb, alb, nrm, _ = _images(case["batch"], case["height"], case["width"], seed)
        h, w = case["height"], case["width"]
        hp, wp = (h + 63) // 64 * 64, (w + 127) // 128 * 128
        y = torch.arange(hp, device="cuda").clamp_max(h - 1)
        x = torch.arange(wp, device="cuda").clamp_max(w - 1)
        params = _weights64()
        with torch.no_grad():
            out = [torch.expm1(_unet64(*(v[b:b + 1][:, y][:, :, x] for v in (rgb, alb, nrm)), params)).clamp_min(0.0)
                   for b in range(case["batch"])]
        return torch.cat(out)[:, :h, :w].contiguous()
    if case["kind"] == "train":
        rgb, alb, nrm, target = _images(case["batch"], case["height"], case["width"], seed)
        params = [(w.requires_grad_(), b.requires_grad_()) for w, b in _weights64()]
        pred = _unet64(rgb, alb, nrm, params)
        loss = (pred - torch.log1p(target.double().clamp_min(0.0))).abs().mean()
        loss.backward()
        grads = [g for w, b in params for g in (w.grad.permute(0, 2, 3, 1).reshape(-1), b.grad)]
        return {"loss": float(loss), "grads": torch.cat(grads)}
    # a path's later vertices depend on every bit of its earlier ones, a query's hit on the
    # rounding of the intersection test, and the rest are whole numbers
    return None
