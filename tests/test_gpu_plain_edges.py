"""The plain f64 form where numbers leave their usual range: rays that are not
numbers, directions far from unit length, path weights that overflow, films of
2^30 pixels.  The oracle runs the reference's loops; pixels are NaN where its
are and equal its to 1e-9 otherwise, but for the samples whose path a last bit
of CUDA's sine or cosine sends another way (at most 0.2%, the bar of the other
plain f64 tests)."""
import math

import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import DeviceScene
from tinypt_b200.scene import Camera, EnvMap, Instance, Material, Mesh, Scene, Sphere, Transform, World
from tests.parity_util import cfg, gpu_film

pytestmark = pytest.mark.gpu

WF, PLAIN = _abi.TPT_MODE_WAVEFRONT_FP32, _abi.TPT_MODE_PLAIN_F64
W, H = 48, 32
INF, NAN = float("inf"), float("nan")


def _same_as_oracle(oracle_mod, scene, spp=4, depth=6, w=W, h=H):
    c = cfg(w, h, spp, depth, PLAIN, seed=3)
    with oracle_mod.OracleScene(scene) as o:
        want, want_w, _, _ = o.render(c, want_sq=True)
    with DeviceScene(scene) as ds:
        (acc, acc_w, _), st = gpu_film(ds, c)
    assert np.array_equal(acc_w, want_w) and st.device_flags == 0
    same = (np.isnan(acc) & np.isnan(want)) | (acc == want) | (np.abs(acc - want) <= 1e-9 * np.maximum(np.abs(want), 1e-12))
    assert (~same.all(axis=1)).mean() <= 1.0 - 0.998 ** spp
    return want


def _spheres(light, aspect):
    """A light as the light-th of five spheres, one of them of a glass that
    refracts into a NaN."""
    mats = [Material.dielectric(INF, (0.1, 0.1, 0.1)), Material.lambert((0.7, 0.5, 0.3)),
            Material.metal((0.8, 0.8, 0.8)), Material.diffuse_light((1.0, 2.0, 3.0))]
    s = Scene(Camera.look_at((0.0, 0.6, 4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 45.0, aspect), World(), mats, None)
    others = [Sphere((-0.8, 0.0, 0.0), 0.5, 0), Sphere((0.8, 0.0, 0.0), 0.5, 1), Sphere((0.0, -100.5, 0.0), 100.0, 2),
              Sphere((0.1, 0.0, -1.0), 0.4, 1)]
    others.insert(light, Sphere((0.0, 0.9, 0.0), 0.3, 3))
    s.world.spheres.extend(others)
    return s


@pytest.mark.parametrize("light", [0, 2, 4])
@pytest.mark.parametrize("aspect", [W / H, NAN])
def test_rays_that_are_not_numbers(gpu, oracle_mod, light, aspect):
    """Every test of the reference's loops lets a NaN pass, so such a ray meets
    the last sphere; mesh hits at a NaN distance do not count."""
    s = _spheres(light, aspect)
    v, f = scenes.displaced_icosphere(1, 0.08, 3, 5)
    s.world.meshes.append(Mesh.from_arrays(v * 0.3, f, 1))
    s.world.instances.append(Instance(0, Transform.translate((0.3, 0.3, 1.0)), None))
    want = _same_as_oracle(oracle_mod, s)
    if math.isnan(aspect):
        assert (want.max() > 0.0) == (light == 4)


def test_directions_of_another_length(gpu, oracle_mod):
    """A mirror ball of radius 1e-11 at 1000 reflects into directions whose
    length is off by a per cent (its normals are).  A hit of a mesh counts at
    dot(p - o, d), a sphere's at its root: a glowing square just
    outside a large sphere may be the closer one from inside."""
    at = np.array([1000.0, 0.0, 0.0])
    u, a = np.array([0.0, 0.0, 1.0]), np.array([1.0, 0.0, 0.0])
    b = np.cross(u, a)
    mats = [Material.metal((0.9, 0.9, 0.9)), Material.lambert((0.9, 0.1, 0.1)), Material.diffuse_light((0.1, 0.1, 0.9))]
    r, d = 1e-11, 2e-4
    s = Scene(Camera.look_at(tuple(at + d * u), tuple(at), (1.0, 0.0, 0.0), math.degrees(0.5 * r / d), W / H),
              World(), mats, None)
    s.world.spheres += [Sphere(tuple(at), r, 0), Sphere(tuple(at - 490.0 * u), 500.0, 1)]
    centre, half = at + 10.1 * u, 5.0
    k = 8  # squares a side, so that the mesh has a tree
    p = np.array([centre + half * ((2 * i / k - 1.0) * a + (2 * j / k - 1.0) * b) for j in range(k + 1) for i in range(k + 1)])
    q = np.array([j * (k + 1) + i for j in range(k) for i in range(k)])
    f = np.concatenate([np.stack([q, q + 1, q + k + 2], 1), np.stack([q, q + k + 2, q + k + 1], 1)])
    s.world.meshes.append(Mesh.from_arrays(p, f, 2))
    s.world.instances.append(Instance(0, Transform.identity(), None))
    want = _same_as_oracle(oracle_mod, s, spp=8, depth=3)
    lit = want[:, 2] > 0.5 * want[:, 2].max()
    assert 0.1 < lit.mean() < 0.9


def _out_of_range(kind):
    v, f = scenes.displaced_icosphere(2, 0.08, 3, 5)
    v = np.array(v)
    at = int(np.argmax(v[:, 2]))  # the vertex nearest the camera
    if kind == "infinite vertex":
        v[at] = [0.1, INF, 0.2]
    elif kind == "nan vertex":
        v[at] = [NAN, NAN, NAN]
    elif kind == "nan in a vertex":
        v[at, 1] = NAN
    elif kind == "vertex at 1e200":
        v[at] = [0.1, 0.2, -1e200]
    mats = [Material.lambert(c) for c in ((0.8, 0.3, 0.2), (0.2, 0.3, 0.8), (0.3, 0.8, 0.3))]
    s = Scene(Camera.look_at((0.0, 0.6, 4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 45.0, W / H), World(), mats, None)
    xf = {"flat transform": Transform.scale((1.0, 0.0, 1.0)), "nan transform": Transform.translate((NAN, 0.0, 0.0)),
          "infinite transform": Transform.translate((0.0, INF, 0.0))}
    s.world.meshes.append(Mesh.from_arrays(v, f, 0))
    s.world.instances.append(Instance(0, Transform.translate((0.1, 0.0, 0.0)), None))
    if kind in xf:
        s.world.instances.append(Instance(0, xf[kind], 1))
    s.world.spheres += [Sphere((1.2, 0.0, 0.0), 0.5, 1), Sphere((-1.4, 0.0, 0.0), 0.5, 2)]
    ball = {"nan sphere": ((NAN, 0.0, 0.0), 0.5), "infinite sphere": ((0.0, INF, 0.0), 0.5), "nan radius": ((0.0, -1.0, 0.0), NAN),
            "infinite radius": ((0.0, -1.0, 0.0), INF), "negative radius": ((0.0, 1.0, 0.0), -0.4)}
    if kind in ball:
        s.world.spheres.insert(1, Sphere(*ball[kind], 2))
    return s


@pytest.mark.parametrize("kind", [
    "usual", "infinite vertex", "nan vertex", "nan in a vertex", "vertex at 1e200", "flat transform", "nan transform",
    "infinite transform", "nan sphere", "infinite sphere", "nan radius", "infinite radius", "negative radius"])
def test_geometry_out_of_range(gpu, oracle_mod, kind):
    _same_as_oracle(oracle_mod, _out_of_range(kind))


@pytest.mark.parametrize("mode", [WF, PLAIN])
@pytest.mark.parametrize("albedos", [(-1e200, -1e200), (1e29, 1e300)])
def test_black_map_with_overflowing_albedo(gpu, mode, albedos):
    """A path weight that overflows times black is a NaN on the general path
    (an unused infinite material selects it), so it is one on the shortcut."""
    c = cfg(W, H, 4, 2, mode, seed=4)
    films = []
    for general in (False, True):
        s = scenes.build_scene(W, H)
        s.env = EnvMap.from_pixels(3, 2, np.zeros((2, 3, 3)))
        s.mats = [Material.lambert((albedos[k % 2], albedos[k % 2], 0.5)) for k in range(len(s.mats))]
        if general:
            s.mats = s.mats + [Material.lambert((INF, 0.0, 0.0))]
        with DeviceScene(s) as ds:
            films.append(gpu_film(ds, c)[0])
    if mode == PLAIN:
        assert np.isnan(films[1][0]).any()
    for a, b in zip(*films):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("w, h", [(1, 70), (5, 4), (7, 33), (8, 5), (9, 33), (33, 12), (200, 5)])
@pytest.mark.parametrize("make", [scenes.build_scene, scenes.sphere_scene])  # each of the form's kernels
def test_pixels_do_not_depend_on_the_tiles(gpu, make, w, h):
    """A film's pixels are handed out by 8 x 4 or, below 8 columns, 1 x 32; a shard
    of its rows with fewer than 4 by 32 x 1.  The shards make up the film, bit for
    bit."""
    step = (h + 2) // 3
    with DeviceScene(make(w, h)) as ds:
        whole = ds.render(cfg(w, h, 4, 4, PLAIN)).acc.reshape(h, w, 3)
        for k in range(step):
            part = ds.render(cfg(w, h, 4, 4, PLAIN, row_begin=k, row_step=step)).acc.reshape(-1, w, 3)
            assert 1 <= len(part) <= 3 and np.array_equal(part, whole[k::step])
    assert whole.min() >= 0.0 and np.count_nonzero(whole.max(axis=2)) > 0


@pytest.mark.parametrize("w, h, depth", [(1 << 30, 1, 0), (1 << 30, 1, 1), (1, 1 << 30, 0), (9, (1 << 30) // 9, 1)])
def test_films_of_2_30_pixels(gpu, w, h, depth):
    """In 8x4 tiles the first has 2^32 pixels, the second 2^33."""
    import torch

    n = w * h
    acc = torch.full((3 * n,), -1.0, dtype=torch.float64, device="cuda")
    acc_w = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()  # the fills run on another stream than the render
    with DeviceScene(scenes.sphere_scene(8, 8)) as ds:
        st = ds.render_device(cfg(w, h, 1, depth, PLAIN), acc.data_ptr(), acc_w.data_ptr())
    torch.cuda.synchronize()
    whole = bool((acc_w == 1.0).all()) and bool((acc >= 0.0).all())  # (not in the assert, which would list the film)
    del acc, acc_w
    torch.cuda.empty_cache()
    assert whole and st.paths == n
