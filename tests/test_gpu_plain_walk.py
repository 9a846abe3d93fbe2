"""The plain f64 form walks the FP32 forms' trees; what it returns must be
what the reference's own walk returns (src/bvh.rs:248-351, src/world.rs:81-121).

Scenes where that depends on the order of the reference's walk or loops --
coincident triangles, spheres and instances of different materials -- and
scenes where the FP32 box tests have the least room: far from the origin,
strongly scaled, flat.  The oracle runs the reference's walk.  Every surface is Lambert, lit by the sky
only, so a wrong primitive changes the pixel's colour; pixels equal the
oracle's to 1e-9 except where a last-bit difference of CUDA's f64 sine or
cosine flips a branch: at most 0.2% of the samples (the bar of the other
plain f64 tests), so 0.998^spp of the pixels are left.
"""
import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import DeviceScene
from tinypt_b200.scene import Camera, Instance, Material, Mesh, Scene, Sphere, Transform, World
from tests.parity_util import cfg, gpu_film

pytestmark = pytest.mark.gpu

PLAIN = _abi.TPT_MODE_PLAIN_F64
COLOURS = [(0.9, 0.1, 0.1), (0.1, 0.9, 0.1), (0.1, 0.1, 0.9), (0.8, 0.8, 0.1)]


def _scene(w, h, eye=(0.0, 0.6, 4.0), at=(0.0, 0.0, 0.0)):
    mats = [Material.lambert(c) for c in COLOURS]
    return Scene(Camera.look_at(eye, at, (0.0, 1.0, 0.0), 45.0, w / h), World(), mats, None)


def _add(s, mesh, *xf, override=None):
    t = Transform.identity()
    for x in xf:
        t = t.compose(x)
    s.world.meshes.append(mesh)
    s.world.instances.append(Instance(len(s.world.meshes) - 1, t, override))


def _sphere_mesh(subdiv, mat):
    v, f = scenes.displaced_icosphere(subdiv, 0.08, 3, 5)
    return v, f, np.full(len(f), mat, dtype=np.int32)


def coincident_triangles(w, h):
    """Every triangle four times, each copy of another material, shuffled."""
    s = _scene(w, h)
    v, f, _ = _sphere_mesh(2, 0)
    m = np.repeat(np.arange(4, dtype=np.int32), len(f))
    order = np.random.default_rng(1).permutation(4 * len(f))
    _add(s, Mesh.from_arrays(v, np.tile(f, (4, 1))[order], m[order]))
    return s


def coincident_spheres(w, h):
    s = _scene(w, h)
    for k in range(4):
        for x in (-1.2, 0.0, 1.2):
            s.world.spheres.append(Sphere((x, 0.0, 0.0), 0.6, (k + int(2 * x)) % 4))
    return s


def coincident_instances(w, h):
    """One mesh four times in the same place, and a sphere touching it."""
    s = _scene(w, h)
    v, f, m = _sphere_mesh(2, 0)
    for k in (2, 0, 3, 1):
        _add(s, Mesh.from_arrays(v, f, m), Transform.translate((0.3, 0.0, 0.0)), override=k)
    s.world.spheres.append(Sphere((-1.0, 0.0, 0.0), 0.5, 1))
    return s


def far_away(w, h):
    c = (3.0e4, -2.0e4, 5.0e4)
    s = _scene(w, h, eye=(c[0], c[1] + 0.6, c[2] + 4.0), at=c)
    _add(s, Mesh.from_arrays(*_sphere_mesh(3, 1)), Transform.translate(c))
    s.world.spheres.append(Sphere((c[0] + 1.2, c[1], c[2]), 0.4, 2))
    s.world.spheres.append(Sphere((c[0], c[1] - 1001.0, c[2]), 1000.0, 0))
    return s


def scaled(w, h):
    s = _scene(w, h)
    big = Mesh.from_arrays(_sphere_mesh(2, 0)[0] * 1.0e4, *_sphere_mesh(2, 0)[1:])
    _add(s, big, Transform.translate((-1.0, 0.0, 0.0)), Transform.scale((1.0e-4, 0.7e-4, 0.6e-4)))
    _add(s, Mesh.from_arrays(*_sphere_mesh(2, 1)), Transform.translate((1.0, 0.0, 0.0)),
         Transform.rotate((1.0, 2.0, 0.5), 40.0), Transform.scale((-0.8, 0.02, 0.9)))
    _add(s, Mesh.from_arrays(np.zeros((3, 3)), np.zeros((0, 3)), 0))  # an empty mesh
    return s


def flat_and_slivers(w, h):
    """Walls seen edge on, and overlapping slivers that crowd towards one edge."""
    s = _scene(w, h, eye=(0.0, 0.0, 4.0))
    for y in (-0.5, 0.0, 0.5):
        _add(s, scenes.unit_rectangle(1), Transform.translate((0.0, y, 0.0)), Transform.rotate((1.0, 0.0, 0.0), 90.0))
    n = 190
    x = -2.0 + 4.0 * 0.5 ** np.arange(n)
    p = np.stack([np.stack([x, 0 * x - 1.0, 0 * x], 1), np.stack([x + 0.3 * (x + 2.0), 0 * x - 1.0, 0 * x], 1),
                  np.stack([x, 0 * x + 1.0, 0 * x], 1)], 1).reshape(-1, 3)
    _add(s, Mesh.from_arrays(p, np.arange(3 * n).reshape(-1, 3), 2), Transform.translate((0.0, 0.0, -1.0)))
    return s


@pytest.mark.parametrize("make, w, h, spp", [
    (coincident_triangles, 48, 32, 4), (coincident_spheres, 47, 31, 4), (coincident_instances, 48, 32, 4),
    (far_away, 48, 32, 4), (scaled, 48, 32, 4), (flat_and_slivers, 48, 32, 4),
    # films that are not whole tiles, of one pixel, and of more pixels than lanes
    (coincident_spheres, 1, 1, 32), (coincident_triangles, 9, 5, 8), (coincident_instances, 301, 203, 1),
    (coincident_triangles, 261, 150, 2),
])
def test_plain_walk_equals_reference_walk(gpu, oracle_mod, make, w, h, spp):
    scene = make(w, h)
    c = cfg(w, h, spp, 6, PLAIN, seed=3)
    with oracle_mod.OracleScene(scene) as o:
        want, want_w, want_sq, _ = o.render(c, want_sq=True)
    with DeviceScene(scene) as ds:
        (acc, acc_w, sq), st = gpu_film(ds, c)
    assert np.array_equal(acc_w, want_w) and st.paths == w * h * spp and st.device_flags == 0
    off = [np.any(np.abs(a - b) > 1e-9 * np.maximum(np.abs(b), 1e-12), axis=1) for a, b in ((acc, want), (sq, want_sq))]
    assert (off[0] | off[1]).mean() <= 1.0 - 0.998 ** spp
