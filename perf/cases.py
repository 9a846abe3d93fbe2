"""Cases by which the renderer's speed is measured.

Each case is one call (or one optimisation step) that a program using this
package makes, through the public entry points: ``DeviceScene.render`` /
``render_device``, ``tpt_render_device_noalloc``, the torch.autograd wrapper
``autodiff.RenderMaterials`` and ``BatchScenes.render``.  Scenes and sizes are
those of the package's own generators, benchmark and tests, or generic ones
of the same ranges (odd film sizes among them).

``prepare`` makes the scene and the handle that a program keeps between
frames; ``run`` is one call and returns the films, images and gradients it
writes.  ``exact`` knows the sample counts of uniform renders; the radiance
sums of a Monte Carlo render have no closed form.
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import math

import numpy as np
import torch

from tinypt_b200 import _abi, autodiff, scenes
from tinypt_b200.render import BatchScenes, DeviceScene
from tinypt_b200.scene import Camera, Material, RenderConfig

_MODE = {"fp32": _abi.TPT_MODE_WAVEFRONT_FP32, "f64": _abi.TPT_MODE_PLAIN_F64}


def listed():
    return [
        # the smallest call: one sample per pixel of the built-in scene, as an
        # interactive preview asks for again and again
        {"name": "preview_64x36", "scene": "default", "call": "device", "mode": "fp32", "width": 64, "height": 36,
         "spp": 1, "depth": 8, "aperture": 0.0},
        # a thumbnail from a program that may not allocate while it renders
        {"name": "noalloc_96x96", "scene": "spheres", "call": "noalloc", "mode": "fp32", "width": 96, "height": 96,
         "spp": 16, "depth": 8},
        # the package's small standard scene (all material kinds, one area
        # light), film in host memory
        {"name": "spheres_256", "scene": "spheres", "call": "host", "mode": "fp32", "width": 256, "height": 256,
         "spp": 64, "depth": 8},
        # an odd film through a lens, second moments for a denoiser
        {"name": "lens_853x479", "scene": "default", "call": "moments", "mode": "fp32", "width": 853, "height": 479,
         "spp": 17, "depth": 8, "aperture": 0.3},
        # an ordinary frame: a mesh of 82K triangles, 200 spheres, env map
        {"name": "frame_960x540", "scene": "mesh_env", "call": "device", "mode": "fp32", "width": 960, "height": 540,
         "spp": 64, "depth": 16, "subdiv": 6, "spheres": 200},
        # the benchmark frame: 1.31M triangles, 200 spheres, 1080p, 256 spp
        {"name": "frame_1920x1080", "scene": "mesh_env", "call": "device", "mode": "fp32", "width": 1920,
         "height": 1080, "spp": 256, "depth": 16, "subdiv": 8, "spheres": 200},
        # one inverse-rendering step: forward image, loss, material gradients
        {"name": "step_512", "scene": "inverse", "call": "step", "mode": "fp32", "width": 512, "height": 512,
         "spp": 64, "depth": 8, "nx": 256, "nz": 512},
        # adaptive sampling of the Cornell box with a GGX mesh and glass
        {"name": "adaptive_480x270", "scene": "cornell", "call": "device", "mode": "fp32", "width": 480,
         "height": 270, "spp": 256, "depth": 32, "n_lat": 128, "n_lon": 256},
        # many small scenes in one call (thumbnails of an asset library)
        {"name": "batch_small_64", "scene": "batch", "call": "batch", "mode": "fp32", "scenes": 64, "tris_lo": 1000,
         "tris_hi": 50000, "res_lo": 32, "res_hi": 96, "spp_lo": 4, "spp_hi": 16, "depth": 12},
        # scenes and films of uneven size in one call
        {"name": "batch_mixed_10", "scene": "batch", "call": "batch", "mode": "fp32", "scenes": 10, "tris_lo": 1000,
         "tris_hi": 200000, "res_lo": 128, "res_hi": 768, "spp_lo": 16, "spp_hi": 128, "depth": 12},
        # the f64 form, which follows the reference draw for draw: the small
        # standard scene, and the kind of frame reference images are made of
        {"name": "f64_spheres_256", "scene": "spheres", "call": "host", "mode": "f64", "width": 256, "height": 256,
         "spp": 64, "depth": 8},
        {"name": "f64_frame_480x270", "scene": "mesh_env", "call": "device", "mode": "f64", "width": 480,
         "height": 270, "spp": 32, "depth": 16, "subdiv": 7, "spheres": 200},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spheres", "default", "mesh_env", "mesh_env", "inverse", "cornell", "batch", "noalloc"])
    if kind == "noalloc":
        return {"scene": rng.choice(["spheres", "default"]), "call": "noalloc", "mode": "fp32",
                "width": _log(rng, 16, 128), "height": _log(rng, 16, 128), "spp": _log(rng, 1, 32),
                "depth": rng.randint(4, 16), "aperture": 0.0}
    if kind in ("spheres", "default"):
        return {"scene": kind, "call": rng.choice(["device", "host", "moments"]), "mode": rng.choice(["fp32", "f64"]),
                "width": _log(rng, 24, 900), "height": _log(rng, 24, 600), "spp": _log(rng, 1, 64),
                "depth": rng.randint(4, 16), "aperture": rng.choice([0.0, 0.0, 0.1, 0.3])}
    if kind == "mesh_env":
        f64 = rng.random() < 0.3
        return {"scene": kind, "call": rng.choice(["device", "host", "moments"]), "mode": "f64" if f64 else "fp32",
                "width": _log(rng, 96, 480 if f64 else 1280), "height": _log(rng, 64, 270 if f64 else 720),
                "spp": _log(rng, 1, 32 if f64 else 128), "depth": rng.randint(4, 16), "subdiv": rng.randint(3, 7),
                "spheres": _log(rng, 10, 200)}
    if kind == "inverse":
        return {"scene": kind, "call": "step", "mode": "fp32", "width": _log(rng, 48, 512),
                "height": _log(rng, 48, 512), "spp": _log(rng, 4, 64), "depth": rng.randint(4, 8),
                "nx": 4 * _log(rng, 8, 64), "nz": 4 * _log(rng, 8, 128)}
    if kind == "cornell":
        f64 = rng.random() < 0.25
        return {"scene": kind, "call": "device", "mode": "f64" if f64 else "fp32",
                "width": _log(rng, 64, 160 if f64 else 480), "height": _log(rng, 36, 90 if f64 else 270),
                "spp": _log(rng, 16, 64 if f64 else 256), "depth": rng.randint(8, 32), "n_lat": 64, "n_lon": 128}
    return {"scene": "batch", "call": "batch", "mode": "fp32", "scenes": _log(rng, 2, 48), "tris_lo": 500,
            "tris_hi": _log(rng, 2000, 50000), "res_lo": 24, "res_hi": _log(rng, 48, 320), "spp_lo": 2,
            "spp_hi": _log(rng, 8, 64), "depth": rng.randint(4, 16)}


# ---- inputs ---------------------------------------------------------------------------------------
def _vary(mats, rng):
    """The scene's materials with other colours: albedos and emissions scaled
    by 0.7 to 1.1 per channel (albedos stay at most 0.97)."""
    out = []
    for m in mats:
        s = rng.uniform(0.7, 1.1, 3)
        top = 1e9 if m.kind in (_abi.TPT_MAT_DIFFUSE_LIGHT, _abi.TPT_MAT_DIELECTRIC) else 0.97
        out.append(Material(m.kind, tuple(float(min(c * k, top)) for c, k in zip(m.rgb, s)), m.param))
    return out


def _scene(case, seed):
    w, h, kind = case["width"], case["height"], case["scene"]
    if kind == "mesh_env":
        return scenes.mesh_env_scene(w, h, subdiv=case["subdiv"], n_spheres=case["spheres"], seed=seed)
    if kind == "cornell":
        s = scenes.cornell_scene(w, h, n_lat=case["n_lat"], n_lon=case["n_lon"], seed=seed)
    elif kind == "default":
        s = scenes.build_scene(w, h)
    else:
        s = scenes.sphere_scene(w, h)
    aperture = case.get("aperture", 0.0)
    if aperture > 0.0:
        c = s.cam
        focus = math.dist(c.eye, c.target)
        s.cam = Camera.look_at_dof(c.eye, c.target, c.up, c.fov_y_deg, c.aspect, focus, aperture)
    s.mats = _vary(s.mats, np.random.default_rng(seed))
    return s


def _config(case, seed):
    cfg = RenderConfig(width=case["width"], height=case["height"], spp=case["spp"], max_bounces=case["depth"],
                       rr_start=3, seed=seed, mode=_MODE[case["mode"]])
    if case["scene"] == "cornell":
        cfg = dataclasses.replace(cfg, adaptive_enabled=True, adaptive_min_spp=8, adaptive_threshold=0.01)
    return cfg


def _batch_configs(case, seed):
    """[(triangles, RenderConfig)]: triangle counts, square films and samples
    log-uniform over the case's ranges, as scenes.batch_workload draws them.
    They belong to the case; the seed picks the scenes and the streams."""
    rng, out = np.random.default_rng(77), []
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))  # noqa: E731
    for k in range(case["scenes"]):
        tris = int(log(case["tris_lo"], case["tris_hi"]))
        res = max(8, int(round(log(case["res_lo"], case["res_hi"]) / 8.0)) * 8)
        spp = int(round(log(case["spp_lo"], case["spp_hi"])))
        out.append((tris, RenderConfig(width=res, height=res, spp=spp, max_bounces=case["depth"], rr_start=3,
                                       seed=64 * seed + k, mode=_MODE["fp32"])))
    return out


def _batch_jobs(case, seed):
    return [(scenes.batch_scene(1000 * seed + k, tris, c.width, c.height), c)
            for k, (tris, c) in enumerate(_batch_configs(case, seed))]


def _f64(n):
    return torch.empty(n, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    st = {"call": case["call"]}
    if case["call"] == "batch":
        work = _batch_jobs(case, seed)
        st["batch"] = BatchScenes([s for s, _ in work])
        px = [c.film_pixels for _, c in work]
        acc, acc_w = _f64(3 * sum(px)), _f64(sum(px))
        jobs, at = [], 0
        for k, (_, c) in enumerate(work):
            jobs.append((k, c, acc.data_ptr() + 24 * at, acc_w.data_ptr() + 8 * at))
            at += px[k]
        st.update(jobs=jobs, acc=acc, acc_w=acc_w)
        return st
    if case["call"] == "step":
        rng = np.random.default_rng(seed)
        s = scenes.inverse_scene(case["width"], case["height"], nx=case["nx"], nz=case["nz"],
                                 params=scenes.inverse_params(seed), seed=seed + 1)
        st["ds"], st["base"] = DeviceScene(s), s.mats
        start = np.clip(autodiff.params_of(s.mats) + rng.normal(0.0, 0.12, (len(s.mats), 4)), 0.05, 0.95)
        st["params"] = torch.tensor(start, requires_grad=True)
        st["target"] = torch.tensor(rng.uniform(0.0, 1.5, (case["height"], case["width"], 3)).astype(np.float32),
                                    device="cuda")
        st["forward"], st["adjoint"] = _config(case, 2 * seed + 1), _config(case, 2 * seed + 2)
        return st
    cfg = _config(case, seed)
    st["ds"], st["cfg"], n = DeviceScene(_scene(case, seed)), cfg, cfg.film_pixels
    if case["call"] == "host":
        st["acc"], st["acc_w"] = np.empty((n, 3)), np.empty((n,))
    else:
        st["acc"], st["acc_w"] = _f64(3 * n), _f64(n)
    if case["call"] == "moments":
        st["acc_sq"] = _f64(3 * n)
    return st


def run(st):
    call = st["call"]
    if call == "batch":
        st["batch"].render(st["jobs"])
    elif call == "step":
        p = st["params"]
        p.grad = None
        img = autodiff.RenderMaterials.apply(p, st["ds"], st["base"], st["forward"], st["adjoint"])
        loss = ((img - st["target"]) ** 2).mean()
        loss.backward()
        return img.detach(), p.grad
    elif call == "host":
        out = st["ds"].render(st["cfg"], acc=st["acc"], acc_w=st["acc_w"])
        return out.acc, out.acc_w
    elif call == "noalloc":
        stats = _abi.tpt_stats()
        _abi.check(_abi.lib().tpt_render_device_noalloc(
            st["ds"]._handle, C.byref(st["cfg"].to_c()), C.c_void_p(st["acc"].data_ptr()),
            C.c_void_p(st["acc_w"].data_ptr()), C.byref(stats)))
    elif call == "moments":
        st["ds"].render_device(st["cfg"], st["acc"].data_ptr(), st["acc_w"].data_ptr(), st["acc_sq"].data_ptr())
        return st["acc"], st["acc_w"], st["acc_sq"]
    else:
        st["ds"].render_device(st["cfg"], st["acc"].data_ptr(), st["acc_w"].data_ptr())
    return st["acc"], st["acc_w"]


def exact(case, seed):
    """Sample counts of uniform renders; nothing else is known in closed form."""
    if case["call"] == "batch":
        cfgs = [c for _, c in _batch_configs(case, seed)]
        return None, torch.cat([torch.full((c.film_pixels,), float(c.spp), dtype=torch.float64) for c in cfgs])
    if case["call"] == "step" or case["scene"] == "cornell":
        return None
    n = case["width"] * case["height"]
    w = torch.full((n,), float(case["spp"]), dtype=torch.float64)
    return (None, w, None) if case["call"] == "moments" else (None, w)


def work(case):
    """Bytes: the scene's triangles (48), spheres (32) and env texels (16) read
    once, the film written once (f64: 32 per pixel, 56 with second moments;
    an image 12).  Operations: per sample two path segments, each a ray and a
    shadow ray through a binary tree over the primitives (two boxes of 24
    operations a level) and 300 operations of shading."""
    if case["call"] == "batch":
        tris = case["scenes"] * math.sqrt(case["tris_lo"] * case["tris_hi"])
        mean = lambda lo, hi: (hi - lo) / math.log(hi / lo) if hi > lo else lo  # noqa: E731  of a log-uniform value
        px = case["scenes"] * mean(case["res_lo"] ** 2, case["res_hi"] ** 2)
        spp, prims, scene = mean(case["spp_lo"], case["spp_hi"]), tris / case["scenes"], 48.0 * tris
    else:
        px, spp = case["width"] * case["height"], case["spp"]
        tris = {"mesh_env": 20 * 4 ** case.get("subdiv", 0), "inverse": 2 * case.get("nx", 0) * case.get("nz", 0),
                "cornell": 2 * case.get("n_lat", 0) * case.get("n_lon", 0) + 36}.get(case["scene"], 2)
        env = {"mesh_env": 1024 * 512, "inverse": 512 * 256}.get(case["scene"], 1)
        spheres = case.get("spheres", 6)
        prims, scene = tris + spheres, 48.0 * tris + 32.0 * spheres + 16.0 * env
        if case["scene"] == "cornell":
            spp = 0.5 * spp  # about half the pixels (the black background) stop at the minimum
    film = {"moments": 56.0, "step": 24.0}.get(case["call"], 32.0) * px
    per_sample = 2.0 * (2.0 * 48.0 * math.log2(prims + 1.0) + 300.0)
    passes = 3.0 if case["call"] == "step" else 1.0  # the adjoint traces the paths again and weighs each vertex
    return {"bytes": scene + film, "flops": passes * px * spp * per_sample}
