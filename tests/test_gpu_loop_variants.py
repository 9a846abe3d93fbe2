"""The bounce loop's variants on small scenes.

By default so small a render runs in one kernel and reaches none of the loop's;
TPT_TAIL_SLOTS=0 (the loop drains itself) and a small handover ask for the loop,
and the iteration count shows that it ran.  Shading register budgets, the
camera-miss fast path and camera culling change no bit of a film, its weights
or its second moments."""
import dataclasses

import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import BatchScenes, DeviceScene
from tests.parity_util import cfg, small_mesh_env_scene

pytestmark = pytest.mark.gpu

WF = _abi.TPT_MODE_WAVEFRONT_FP32
HANDOVER = ["0", "1024"]


@pytest.fixture(autouse=True)
def default_schedule(monkeypatch):
    for k in ("TPT_TASK_SPP", "TPT_POOL", "TPT_CAMERA_FAST", "TPT_SHADE_CTAS", "TPT_MAX_PART_TASKS", "TPT_SHADE_SORT",
              "TPT_WAVEFRONT_HOST_LOOP", "TPT_QUEUE_ORDER", "TPT_QUEUE_DIV", "TPT_SKY_CULL", "TPT_TAIL_SLOTS"):
        monkeypatch.delenv(k, raising=False)


def _film(ds, c, loop=True):
    import torch

    n = c.film_pixels
    film = [torch.full((k * n,), -1.0, dtype=torch.float64, device="cuda") for k in (3, 1, 3)]
    torch.cuda.synchronize()
    st = ds.render_device(c, *(f.data_ptr() for f in film))
    assert (st.iterations > 0) == loop and st.paths == n * c.spp
    return [f.cpu().numpy() for f in film], st


def _same(films):
    for other in films[1:]:
        for a, b in zip(films[0], other):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("tail", HANDOVER)
@pytest.mark.parametrize("make, size, depth", [
    (lambda: scenes.mesh_env_scene(64, 48, subdiv=4, n_spheres=30, env_w=64, env_h=32), (64, 48, 16), 8),
    (lambda: scenes.cornell_scene(48, 40, n_lat=12, n_lon=24), (48, 40, 16), 24),
    (lambda: scenes.sphere_scene(64, 48), (64, 48, 16), 8),
])
def test_shading_budgets_agree(gpu, monkeypatch, tail, make, size, depth):
    c = cfg(*size, depth, WF)
    with DeviceScene(make()) as ds:
        films = [_film(ds, c, loop=False)[0]]
        monkeypatch.setenv("TPT_TAIL_SLOTS", tail)
        for ctas in ("8", "6", "4"):
            monkeypatch.setenv("TPT_SHADE_CTAS", ctas)
            films.append(_film(ds, c)[0])
    _same(films)


@pytest.mark.parametrize("tail", HANDOVER)
def test_camera_miss_fast_path_agrees(gpu, monkeypatch, tail):
    c = cfg(96, 54, 24, 16, WF)
    monkeypatch.setenv("TPT_TASK_SPP", "8")
    monkeypatch.setenv("TPT_TAIL_SLOTS", tail)
    films = []
    with DeviceScene(small_mesh_env_scene()) as ds:
        for fast in ("1", "0"):
            monkeypatch.setenv("TPT_CAMERA_FAST", fast)
            for cull in ("0", "1"):
                monkeypatch.setenv("TPT_SKY_CULL", cull)
                films.append(_film(ds, c)[0])
    _same(films)


@pytest.mark.parametrize("tail", HANDOVER)
@pytest.mark.parametrize("schedule", ["one_task", "task8", "long_tasks", "row_shard"])
def test_culling_agrees(gpu, monkeypatch, tail, schedule):
    c = cfg(96, 54, 96 if schedule == "long_tasks" else 16, 8, WF)
    if schedule == "row_shard":
        c = cfg(96, 54, 16, 8, WF, row_begin=1, row_step=3)
    else:
        monkeypatch.setenv("TPT_TASK_SPP", {"one_task": "16", "task8": "8", "long_tasks": "48"}[schedule])
    with DeviceScene(small_mesh_env_scene(96, 54)) as ds:
        films = [_film(ds, c, loop=False)[0]]
        monkeypatch.setenv("TPT_TAIL_SLOTS", tail)
        for cull in ("1", "0"):
            monkeypatch.setenv("TPT_SKY_CULL", cull)
            film, st = _film(ds, c)
            films.append(film)
            assert (st.sky_samples > 0.2 * st.paths) == (cull == "1")
    _same(films)


def test_batch_variants_agree(gpu, monkeypatch):
    """Shading budgets, culling and the handover in batch renders; one job
    through a lens, one a row shard."""
    import torch

    work = scenes.batch_workload(5, seed=3, tri_range=(500, 30_000), res_range=(24, 80), spp_range=(4, 40), max_depth=8)
    cfgs = [(k, c) for k, (_, c) in enumerate(work)]
    cfgs.append((0, dataclasses.replace(work[0][1], width=40, height=30, spp=20, seed=99, row_begin=1, row_step=2)))
    lens = dataclasses.replace(work[1][0])
    cam = lens.cam
    lens.cam = scenes.Camera.look_at_dof(cam.eye, cam.target, cam.up, cam.fov_y_deg, cam.aspect, 6.0, 0.2)
    cfgs.append((len(work), work[1][1]))
    out = []
    with BatchScenes([s for s, _ in work] + [lens]) as bs:
        for tail in (None, *HANDOVER):
            if tail:
                monkeypatch.setenv("TPT_TAIL_SLOTS", tail)
            for ctas, cull in ((8, "1"), (4, "1"), (8, "0")):
                monkeypatch.setenv("TPT_SKY_CULL", cull)
                films = [(torch.full((3 * c.film_pixels,), -1.0, dtype=torch.float64, device="cuda"),
                          torch.full((c.film_pixels,), -1.0, dtype=torch.float64, device="cuda")) for _, c in cfgs]
                torch.cuda.synchronize()
                st = bs.render([(k, c, a.data_ptr(), w.data_ptr()) for (k, c), (a, w) in zip(cfgs, films)],
                               tuning=(0, 4, 0, ctas))
                assert (st.iterations > 0) == (tail is not None) and (st.sky_samples > 0) == (cull == "1")
                out.append([x.cpu() for f in films for x in f])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert torch.equal(a, b)
