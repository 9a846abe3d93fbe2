"""The plain f64 form's kernels beside the general one.

Scenes of spheres alone run in a kernel of their own; a triangle that no ray
meets sends the same render to the general kernel, whose film must be the same
bit for bit.  One bounce among triangles ends its samples earlier in the
general kernel; those films are compared with the oracle."""
import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import DeviceScene
from tinypt_b200.scene import Camera, EnvMap, Instance, Material, Mesh, RenderConfig, Scene, Sphere, Transform, World
from tests.parity_util import small_mesh_env_scene
from tests.test_gpu_plain_walk import coincident_spheres

pytestmark = pytest.mark.gpu

PLAIN = _abi.TPT_MODE_PLAIN_F64


def _empty(w, h, env=None):
    return Scene(Camera.look_at((0.0, 0.0, 1.5), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 45.0, w / h), World(), [], env)


def _spheres(w, h, n, env):
    """n spheres of every material, one of them a light."""
    rng = np.random.default_rng(n)
    s = _empty(w, h, env)
    s.mats = [Material.lambert((0.7, 0.5, 0.3)), Material.metal((0.8, 0.8, 0.8)), Material.dielectric(1.5, (0.1, 0.2, 0.3)),
              Material.ggx((0.8, 0.6, 0.4), 0.2), Material.subsurface((0.8, 0.7, 0.6), 0.05), Material.diffuse_light((8.0, 7.0, 5.0))]
    for k in range(n):
        s.world.spheres.append(Sphere(tuple(rng.uniform((-2.0, -1.5, -4.0), (2.0, 1.5, -0.5))), float(rng.uniform(0.05, 0.5)), k % 6))
    return s


def _out_of_sight(s):
    """A triangle of 1e-30 that no ray comes near."""
    p = np.array([[0.0, 0.0, 0.0], [1e-30, 0.0, 0.0], [0.0, 1e-30, 0.0]])
    s.mats = list(s.mats) or [Material.lambert((0.5, 0.5, 0.5))]
    s.world.meshes.append(Mesh.from_arrays(p, np.array([[0, 1, 2]]), 0))
    s.world.instances.append(Instance(len(s.world.meshes) - 1, Transform.translate((0.0, 1e6, 0.0)), None))
    return s


def _film(s, c):
    import torch

    n = c.film_pixels
    film = [torch.full((k * n,), -1.0, dtype=torch.float64, device="cuda") for k in (3, 1, 3)]
    torch.cuda.synchronize()
    with DeviceScene(s) as ds:
        st = ds.render_device(c, *(f.data_ptr() for f in film))
    return [f.cpu().numpy() for f in film], st


def _cfg(w, h, spp, depth, rr=3, **kw):
    return RenderConfig(width=w, height=h, spp=spp, max_bounces=depth, rr_start=rr, seed=5, mode=PLAIN, **kw)


@pytest.mark.parametrize("make, c", [
    (lambda: scenes.build_scene(61, 37), _cfg(61, 37, 5, 1)),
    (lambda: scenes.build_scene(61, 37), _cfg(61, 37, 5, 1, rr=0)),
    (lambda: scenes.build_scene(61, 37), _cfg(61, 37, 3, 0)),
    (lambda: scenes.build_scene(64, 36), _cfg(64, 36, 8, 1, row_begin=1, row_step=3)),
    (lambda: scenes.build_scene(48, 32), _cfg(48, 32, 64, 1, adaptive_enabled=True, adaptive_min_spp=4, adaptive_threshold=0.3)),
    (lambda: scenes.build_scene(1, 1), _cfg(1, 1, 7, 1)),
    (lambda: scenes.build_scene(301, 203), _cfg(301, 203, 2, 1)),
    (lambda: scenes.build_scene(61, 37), _cfg(61, 37, 5, 8)),
    (lambda: scenes.build_scene(61, 37), _cfg(61, 37, 5, 20, rr=0)),
    (lambda: _spheres(61, 37, 1, scenes.sky_env(16, 8)), _cfg(61, 37, 5, 8)),
    (lambda: _spheres(61, 37, 60, scenes.sky_env(17, 9)), _cfg(61, 37, 5, 8, rr=1)),
    (lambda: _spheres(61, 37, 255, None), _cfg(61, 37, 5, 8)),
    (lambda: _spheres(61, 37, 60, EnvMap.constant((0.0, 0.0, 0.0))), _cfg(61, 37, 5, 8)),
    (lambda: coincident_spheres(47, 31), _cfg(47, 31, 4, 6)),
    (lambda: _empty(61, 37), _cfg(61, 37, 5, 8)),
    (lambda: _empty(61, 37, scenes.sky_env(16, 8)), _cfg(61, 37, 5, 8)),
    (lambda: _empty(5, 3, scenes.sky_env(16, 8)), _cfg(5, 3, 5, 1)),
])
def test_own_kernel_equals_the_general_one(gpu, make, c):
    (a, st_a), (b, st_b) = _film(make(), c), _film(_out_of_sight(make()), c)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert a[0].min() >= 0.0 and (c.max_bounces == 0 or a[0].max() > 0.0)
    assert (st_a.paths, st_a.rays_closest, st_a.rays_shadow) == (st_b.paths, st_b.rays_closest, st_b.rays_shadow)


@pytest.mark.parametrize("make", [
    lambda: scenes.sphere_scene(96, 64), lambda: small_mesh_env_scene(96, 64),
    lambda: scenes.cornell_scene(96, 64, n_lat=8, n_lon=16), lambda: scenes.build_scene(96, 64),
])
@pytest.mark.parametrize("rr", [0, 3])
def test_one_bounce_equals_the_reference(gpu, oracle_mod, make, rr):
    """Pixels equal the oracle's to 1e-9 but for the samples that a last bit of
    CUDA's f64 sine or cosine sends another way: at most 0.2% of them (the bar of
    the other plain f64 tests) and, of the pixels a shadow ray then misses or
    meets, four standard deviations."""
    c = _cfg(96, 64, 6, 1, rr=rr)
    with oracle_mod.OracleScene(make()) as o:
        want, want_w, want_sq, _ = o.render(c, want_sq=True)
    (acc, acc_w, sq), st = _film(make(), c)
    assert np.array_equal(acc_w, want_w) and st.device_flags == 0
    off = [np.any(np.abs(x.reshape(-1, 3) - y) > 1e-9 * np.maximum(np.abs(y), 1e-12), axis=1) for x, y in ((acc, want), (sq, want_sq))]
    p, n = 1.0 - 0.998 ** c.spp, c.film_pixels
    assert (off[0] | off[1]).mean() <= p + 4.0 * (p * (1.0 - p) / n) ** 0.5
