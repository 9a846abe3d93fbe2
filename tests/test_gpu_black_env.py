"""A black env map (XML scenes carry one) is not looked up: its samples only
take their draws.  A scene with an unused infinite material keeps the general
path, whose film is the same bit for bit."""
import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import DeviceScene
from tinypt_b200.scene import EnvMap, Material
from tests.parity_util import cfg, gpu_film

pytestmark = pytest.mark.gpu

WF, PLAIN = _abi.TPT_MODE_WAVEFRONT_FP32, _abi.TPT_MODE_PLAIN_F64


@pytest.mark.parametrize("mode", [WF, PLAIN])
@pytest.mark.parametrize("name", ["spheres", "cornell", "spheres_3x2_map", "spheres_loop"])
def test_black_map_is_the_general_path(gpu, monkeypatch, mode, name):
    if name == "spheres_loop":
        monkeypatch.setenv("TPT_TAIL_SLOTS", "0")
    make = {"cornell": lambda: scenes.cornell_scene(40, 24, n_lat=8, n_lon=16)}.get(name, lambda: scenes.sphere_scene(40, 24))
    c = cfg(40, 24, 6, 8, mode, seed=4)
    films = []
    for general in (False, True):
        s = make()
        if name == "spheres_3x2_map":
            s.env = EnvMap.from_pixels(3, 2, np.zeros((2, 3, 3)))
        if general:
            s.mats = s.mats + [Material.lambert((float("inf"), 0.0, 0.0))]
        with DeviceScene(s) as ds:
            films.append(gpu_film(ds, c))
    (a, st_a), (b, st_b) = films
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert a[0].max() > 0.0 and st_a.rays_closest == st_b.rays_closest and st_a.rays_shadow == st_b.rays_shadow
