"""The f64 form's env-map samples start from brackets too, made over CDFs that
are not normalised.  The oracle searches the whole CDF, as the reference does
(src/env.rs:124-152): a wrong bracket draws another texel and changes the pixel.
Maps of sizes around the tables' powers of two, with black rows and columns,
single bright texels, long flat runs, weights from 1e-300 to 1e300."""
import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import DeviceScene
from tinypt_b200.scene import EnvMap, Material
from tests.parity_util import cfg, gpu_film

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
    elif kind == "tiny":
        img *= 1e-300
    elif kind == "huge":
        img *= 1e300
    return EnvMap.from_pixels(w, h, img)


@pytest.mark.parametrize("kind", ["noise", "spike", "holes", "flat", "tiny", "huge"])
@pytest.mark.parametrize("w, h", [(1, 1), (2, 1), (3, 2), (16, 8), (17, 9), (255, 1), (1023, 5), (1100, 3), (4, 1030)])
def test_f64_samples_are_the_reference_s(gpu, oracle_mod, w, h, kind):
    """Pixels equal the oracle's to 1e-9 but for the samples that a last bit of
    CUDA's f64 sine or cosine sends another way: at most 0.2% of them (the bar of
    the other plain f64 tests) and four standard deviations.  Lambert spheres, whose
    density is smooth in the sampled direction, at one bounce: all draws before the
    first contribution are exact."""
    s = scenes.build_scene(64, 36)
    s.mats = [Material.lambert((0.7, 0.6, 0.5)) for _ in s.mats]
    s.env = _map(w, h, kind)
    c = cfg(64, 36, 4, 1, _abi.TPT_MODE_PLAIN_F64, seed=11)
    with oracle_mod.OracleScene(s) as o:
        want, want_w, _, _ = o.render(c, want_sq=True)
    with DeviceScene(s) as ds:
        (acc, acc_w, _), st = gpu_film(ds, c)
    assert np.array_equal(acc_w, want_w) and st.device_flags == 0 and np.count_nonzero(want) > 0
    off = np.any(np.abs(acc - want) > 1e-9 * np.maximum(np.abs(want), 1e-300), axis=1)
    p, n = 1.0 - 0.998 ** c.spp, c.film_pixels
    assert off.mean() <= p + 4.0 * (p * (1.0 - p) / n) ** 0.5
