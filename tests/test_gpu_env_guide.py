"""Env-map samples start their CDF searches from a table of brackets in single
renders; batch renders search the whole CDF.  The sample is the same, so the
films are, bit for bit: maps of sizes around the table's powers of two, with
black rows and columns, single bright texels and long flat runs."""
import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import BatchScenes, DeviceScene
from tinypt_b200.scene import EnvMap
from tests.parity_util import cfg

pytestmark = pytest.mark.gpu


def _map(w, h, kind):
    rng = np.random.default_rng(w * 1000 + h)
    img = rng.uniform(0.0, 1.0, (h, w, 3)) ** 4
    if kind == "spike":
        img *= 1e-6
        img[h // 2, w // 3] = 1e5
    elif kind == "holes":
        img[::2] = 0.0
        img[:, w // 4: 3 * w // 4] = 0.0
        img[-1, -1] = 1.0
    elif kind == "flat":
        img[:] = 0.5
    return EnvMap.from_pixels(w, h, img)


@pytest.mark.parametrize("kind", ["noise", "spike", "holes", "flat"])
@pytest.mark.parametrize("w, h", [(1, 1), (2, 1), (3, 2), (16, 8), (17, 9), (255, 1), (1023, 5), (1100, 3), (4, 1030)])
def test_guided_search_draws_the_same_samples(gpu, monkeypatch, w, h, kind):
    import torch

    monkeypatch.setenv("TPT_TASK_SPP", "4")
    scene = scenes.build_scene(32, 18)
    scene.env = _map(w, h, kind)
    c = cfg(32, 18, 8, 4, _abi.TPT_MODE_WAVEFRONT_FP32)
    n = c.film_pixels
    films = [(torch.zeros(3 * n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda"))
             for _ in range(2)]
    with DeviceScene(scene) as ds:
        ds.render_device(c, films[0][0].data_ptr(), films[0][1].data_ptr())
    with BatchScenes([scene]) as bs:
        bs.render([(0, c, films[1][0].data_ptr(), films[1][1].data_ptr())])
    torch.cuda.synchronize()
    assert torch.equal(films[0][0], films[1][0]) and torch.equal(films[0][1], films[1][1])
