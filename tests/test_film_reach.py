"""The gather of the film filters looks only at the source pixels a footprint can
reach (footprint_reach): against every sample of the tile, on the CPU, for filter
sizes around whole and half pixels and samples on the edges of their pixels."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cadise_gb300 import abi

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


@pytest.fixture(scope="module")
def khc(tmp_path_factory):
    from cadise_gb300.native_build import CXX_FLAGS, _cuda_include
    d = tmp_path_factory.mktemp("reach")
    so = str(d / "khc.so")
    csrc = os.path.join(ROOT, "cadise_gb300", "csrc")
    subprocess.check_call(["g++"] + CXX_FLAGS + ["-shared", "-w", "-I", os.path.join(ROOT, "include"), "-I", _cuda_include(),
                                                 os.path.join(ROOT, "tests", "native", "kernel_host_check.cpp")] +
                          [os.path.join(csrc, f) for f in ("scene_build.cpp", "bvh_build.cpp", "tie_order.cpp")] + ["-o", so])
    L = C.CDLL(so)
    L.khc_filter_gather.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_uint32, C.c_void_p, C.c_void_p, C.c_void_p]
    return L


@pytest.mark.parametrize("size", [0.5, 1.0, 1.3, 2.0, 2.9999998, 3.0, 3.0000002, 4.0, 5.7, 9.0])
@pytest.mark.parametrize("shape", [(37, 23), (1500, 3)])
def test_gather_reaches_every_sample(khc, size, shape):
    W, H = shape
    count = 3
    rng = np.random.default_rng(int(size * 1000) + W)
    jit = rng.random((count, H, W, 2)).astype(np.float32)
    jit[0, ::2] = 0.0
    jit[1, ::2] = np.float32(1.0 - 2.0 ** -24)  # rounds up to the next pixel's edge from x = 1 on
    jit[2, ::3] = 0.5
    xy = np.empty_like(jit)
    xy[..., 0] = np.arange(W, dtype=np.float32)[None, None, :] + jit[..., 0]
    xy[..., 1] = np.arange(H, dtype=np.float32)[None, :, None] + jit[..., 1]
    rgb = rng.random((count, H, W, 3)).astype(np.float32)
    film = np.zeros((H, W, 7))
    f = abi.cgpu_film_filter(type=0, width=size, height=size)
    assert khc.khc_filter_gather(C.addressof(f), W, H, count, xy.ctypes.data, rgb.ctypes.data, film.ctypes.data) == 0
    # every sample's own footprint, in the reference's FP32 steps (filmTile.cpp:36-66)
    half = np.float32(size) * np.float32(0.5)
    ref = np.zeros((H, W))
    for axis_tile in [(ty, tx) for ty in range(0, H, 16) for tx in range(0, W, 16)]:
        ty, tx = axis_tile
        ty1, tx1 = min(ty + 16, H), min(tx + 16, W)
        p = xy[:, ty:ty1, tx:tx1].reshape(-1, 2)

        def span(v, t0, t1):
            lo = np.maximum(v - half, np.float32(t0)) - np.float32(0.5)
            hi = np.minimum(v + half, np.float32(t1)) - np.float32(0.5)
            return np.ceil(lo).astype(int), (np.floor(hi) + np.float32(1.0)).astype(int)

        xa, xb = span(p[:, 0], tx, tx1)
        ya, yb = span(p[:, 1], ty, ty1)
        for i in range(len(p)):
            ref[ya[i]:yb[i], xa[i]:xb[i]] += 1.0
    assert np.array_equal(film[..., 6], ref)
