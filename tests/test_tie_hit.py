"""What follows the persistent passes' closest hits (tie_hit), on the CPU: a ray
that met several records within the tie window gets the record of the traversal
from its origin, and is never turned into a miss."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cadise_gb300 import abi, scenes

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
CSRC = os.path.join(ROOT, "cadise_gb300", "csrc")


@pytest.fixture(scope="module")
def tc(tmp_path_factory):
    from cadise_gb300.native_build import CXX_FLAGS, _cuda_include
    so = str(tmp_path_factory.mktemp("tc") / "tie_check.so")
    srcs = [os.path.join(ROOT, "tests", "native", "tie_check.cpp")]
    srcs += [os.path.join(CSRC, f) for f in ("scene_build.cpp", "bvh_build.cpp", "tie_order.cpp")]
    subprocess.check_call(["g++"] + CXX_FLAGS + ["-shared", "-I", os.path.join(ROOT, "include"), "-I", _cuda_include()] +
                          srcs + ["-o", so])
    L = C.CDLL(so)
    L.tc_create.restype = C.c_void_p
    L.tc_create.argtypes = [C.c_void_p, C.c_char_p, C.c_int]
    L.tc_destroy.argtypes = [C.c_void_p]
    L.tc_several.argtypes = [C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p, C.c_void_p, C.c_void_p]
    return L


def box_with(positions):
    s = scenes.cornell_box(8, 8, 1, 2)
    s.primitives = [p for p in s.primitives if not isinstance(p, scenes.TriangleMesh)]
    s.primitives.append(scenes.TriangleMesh(name="mesh", material=s.materials[1].name, positions=positions))
    return abi.flatten(s)


@pytest.mark.parametrize("width", [1e-3, 1e-4])
@pytest.mark.parametrize("graze", [1e-1, 1e-2, 1e-4])
def test_several_records_within_the_window(tc, width, graze):
    """Three copies of each of 300 slivers along the axes, 400 long, met at a
    grazing angle: the rounding of their narrow side moves a hit by more than
    the window along the ray, out of the interval of the sliver's own box."""
    rng = np.random.default_rng(0)
    n, m = 300, 6000
    axis = rng.integers(0, 3, n)
    d = np.eye(3)[axis]
    side = np.eye(3)[(axis + 1) % 3] * np.where(rng.random(n) < 0.5, 1, -1)[:, None]
    a = np.array([278, 273, 280.0]) + rng.uniform(-260, 260, (n, 3))
    tri = np.stack([a - 200 * d, a + 200 * d, a + width * side], 1)
    flat = box_with(np.concatenate([tri] * 3).astype(np.float32))
    k = rng.integers(0, n, m)
    target = (tri.astype(np.float32)[k] * rng.dirichlet([1, 1, 1], m)[:, :, None]).sum(1)
    dirs = d[k] * np.where(rng.random(m) < 0.5, 1, -1)[:, None] + graze * rng.normal(0, 1, (m, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    rays = np.zeros((m, 8), np.float32)
    rays[:, :3] = target - dirs * rng.uniform(1, 300, (m, 1))
    rays[:, 4:7], rays[:, 3], rays[:, 7] = dirs, 1e-3, 3.4e38
    err = C.create_string_buffer(512)
    scene = tc.tc_create(C.addressof(flat.desc), err, 512)
    assert scene, err.value
    held, resolved, general = np.zeros((m, 2), np.int32), np.zeros(m, np.int32), np.zeros(m, np.int32)
    tc.tc_several(scene, rays.ctypes.data, m, held.ctypes.data, resolved.ctypes.data, general.ctypes.data)
    tc.tc_destroy(scene)
    several = held[:, 1] > 2
    assert several.sum() > m // 4
    assert np.all(resolved[several] >= 0)
    assert np.array_equal(resolved[several], general[several])
