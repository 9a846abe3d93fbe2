"""Env-map lookups of the f64 form for directions that are not numbers.

An infinite index of refraction (a scene file's `ext_ior` of 0 gives one) or
GGX alpha turns a ray's direction into a NaN.  The reference's `as usize` takes
texel 0 then (src/env.rs:92-121) and the pixel becomes a NaN; no index may
leave the map."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tinypt_b200 import _abi, scenes
from tinypt_b200.render import DeviceScene
from tinypt_b200.scene import Camera, Instance, Material, Mesh, Scene, Transform, World
from tests.parity_util import cfg, gpu_film

CSRC = Path(__file__).resolve().parent.parent / "tinypt_b200" / "csrc"


def test_texel_index_holds_every_double_to_its_axis(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    src = tmp_path / "t.cpp"
    src.write_text("""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <limits>
#include "texel.hpp"
int main() {
    const double nan = std::numeric_limits<double>::quiet_NaN(), inf = std::numeric_limits<double>::infinity();
    const int sizes[] = {0, 1, 2, 3, 512, 1024, 65536};
    for (int n : sizes)
        for (double f : {nan, -nan, -inf, -1e300, -1.0, -0.0, 0.0, 0.5, 1.0, std::nextafter((double)n, 0.0), (double)n,
                         std::nextafter((double)n, inf), n + 1.0, 3e9, 1e300, inf}) {
            const double g = std::floor(f);
            const int want = !(g > 0.0) ? 0 : (g > (double)n ? n : (int)g);
            if (tpt::texel_index(f, n) != want) { std::printf("%d %g\\n", n, f); return 1; }
        }
    return 0;
}
""")
    exe = tmp_path / "t"
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _scene(w, h):
    mats = [Material.dielectric(float("inf"), (0.1, 0.1, 0.1)), Material.lambert((0.7, 0.5, 0.3)),
            Material.ggx((0.8, 0.8, 0.8), float("inf"))]
    s = Scene(Camera.look_at((0.0, 0.6, 4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 45.0, w / h), World(), mats,
              scenes.sky_env(16, 8))
    v, f = scenes.displaced_icosphere(2, 0.08, 3, 5)
    for k, x in enumerate((-1.2, 0.0, 1.2)):
        s.world.meshes.append(Mesh.from_arrays(v * 0.6, f, np.full(len(f), k, dtype=np.int32)))
        s.world.instances.append(Instance(k, Transform.translate((x, 0.0, 0.0)), None))
    return s


@pytest.mark.gpu
def test_nan_directions_give_the_reference_s_pixels(gpu, oracle_mod):
    """Pixels are NaN where the oracle's are; the others equal its to 1e-9, but
    for the samples whose path a last bit of CUDA's sine or cosine sends
    another way (at most 0.2%, the bar of the other plain f64 tests)."""
    w, h, spp = 48, 32, 4
    scene, c = _scene(w, h), cfg(w, h, spp, 6, _abi.TPT_MODE_PLAIN_F64, seed=3)
    with oracle_mod.OracleScene(scene) as o:
        want, want_w, _, _ = o.render(c, want_sq=True)
    assert 0.02 < np.isnan(want).any(axis=1).mean() < 0.5
    with DeviceScene(scene) as ds:
        (acc, acc_w, _), st = gpu_film(ds, c)
    assert np.array_equal(acc_w, want_w) and st.device_flags == 0
    same = (np.isnan(acc) & np.isnan(want)) | (np.abs(acc - want) <= 1e-9 * np.maximum(np.abs(want), 1e-12))
    assert (~same.all(axis=1)).mean() <= 1.0 - 0.998 ** spp
