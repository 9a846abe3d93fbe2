"""Small FP32 renders run in one kernel (k_paths) instead of the bounce loop.
Its steps and their order are the loop's, so films, sample counts, second
moments and ray counts are the loop's bit for bit (TPT_TAIL_SLOTS=0 asks for
the loop); culled pixels are the same ones."""
import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import BatchScenes, DeviceScene
from tinypt_b200.scene import Camera
from tests.parity_util import cfg, small_mesh_env_scene

pytestmark = pytest.mark.gpu

WF = _abi.TPT_MODE_WAVEFRONT_FP32


@pytest.fixture(autouse=True)
def default_schedule(monkeypatch):
    for k in ("TPT_TASK_SPP", "TPT_POOL", "TPT_CAMERA_FAST", "TPT_SHADE_CTAS", "TPT_MAX_PART_TASKS",
              "TPT_WAVEFRONT_HOST_LOOP", "TPT_QUEUE_ORDER", "TPT_QUEUE_DIV", "TPT_SKY_CULL", "TPT_TAIL_SLOTS"):
        monkeypatch.delenv(k, raising=False)


def _lens(w, h):
    s = scenes.build_scene(w, h)
    s.cam = Camera.look_at_dof(s.cam.eye, s.cam.target, s.cam.up, 40.0, w / h, 4.0, 0.3)
    return s


CASES = {
    # films of one pixel, of fewer and of more paths than lanes in flight
    "one_pixel": (lambda: scenes.sphere_scene(1, 1), cfg(1, 1, 3, 8, WF), None),
    "odd_film": (lambda: scenes.sphere_scene(61, 37), cfg(61, 37, 5, 8, WF), None),
    "many_paths": (lambda: small_mesh_env_scene(96, 54), cfg(301, 203, 3, 16, WF), None),
    # tasks of several samples, the last one short; one task per pixel
    "task8": (lambda: small_mesh_env_scene(96, 54), cfg(96, 54, 19, 16, WF), "8"),
    "one_task": (lambda: scenes.gradcheck_scene(64, 64), cfg(64, 64, 16, 6, WF), "16"),
    "lens": (lambda: _lens(64, 36), cfg(64, 36, 8, 8, WF), None),
    "no_bounce": (lambda: scenes.build_scene(64, 36), cfg(64, 36, 4, 0, WF), None),
    "row_shard": (lambda: small_mesh_env_scene(96, 54), cfg(96, 54, 8, 8, WF, row_begin=1, row_step=3), "4"),
    "adaptive": (lambda: scenes.sphere_scene(48, 32),
                 cfg(48, 32, 64, 8, WF, adaptive_enabled=1, adaptive_min_spp=8, adaptive_threshold=0.05), None),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_one_kernel_equals_the_loop(gpu, monkeypatch, name):
    make, c, task_spp = CASES[name]
    if task_spp:
        monkeypatch.setenv("TPT_TASK_SPP", task_spp)
    got = {}
    import torch

    with DeviceScene(make()) as ds:
        for tail in (None, "0"):
            if tail:
                monkeypatch.setenv("TPT_TAIL_SLOTS", tail)
            n = c.film_pixels
            film = [torch.full((k * n,), -1.0, dtype=torch.float64, device="cuda") for k in (3, 1, 3)]
            st = ds.render_device(c, *(f.data_ptr() for f in film))
            torch.cuda.synchronize()
            got[tail] = ([f.cpu().numpy() for f in film], st)
    (one, st1), (loop, st0) = got[None], got["0"]
    assert st1.iterations == 0 < st0.iterations
    for a, b in zip(one, loop):
        assert np.array_equal(a, b)
    assert (st1.paths, st1.rays_shadow, st1.sky_samples) == (st0.paths, st0.rays_shadow, st0.sky_samples)
    assert st1.rays_closest == st0.rays_closest


def test_one_kernel_batch_equals_the_loop(gpu, monkeypatch):
    import torch

    work = scenes.batch_workload(6, seed=9, tri_range=(200, 5000), res_range=(8, 56), spp_range=(1, 21), max_depth=8)

    def render():
        films = [(torch.zeros(3 * c.film_pixels, dtype=torch.float64, device="cuda"),
                  torch.zeros(c.film_pixels, dtype=torch.float64, device="cuda")) for _, c in work]
        with BatchScenes([s for s, _ in work]) as bs:
            st = bs.render([(k, c, a.data_ptr(), w.data_ptr()) for k, ((_, c), (a, w)) in enumerate(zip(work, films))])
        return films, st

    one, st1 = render()
    monkeypatch.setenv("TPT_TAIL_SLOTS", "0")
    loop, st0 = render()
    assert st1.iterations == 0 < st0.iterations
    assert (st1.paths, st1.rays_shadow, st1.sky_samples) == (st0.paths, st0.rays_shadow, st0.sky_samples)
    for (a1, w1), (a0, w0) in zip(one, loop):
        assert torch.equal(w1, w0) and torch.equal(a1, a0)
