"""Device buffers hold what their kernels use: a closest-hit pass has at most one
ray a path, and so have its tie queue and its sort."""
import ctypes as C
import os
import subprocess

import pytest

import cadise_gb300 as cg
from cadise_gb300 import scenes

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


@pytest.fixture(scope="module")
def ly(tmp_path_factory):
    from cadise_gb300.native_build import CXX_FLAGS, _cuda_include
    so = str(tmp_path_factory.mktemp("ly") / "layout_check.so")
    subprocess.check_call(["g++"] + CXX_FLAGS + ["-shared", "-I", os.path.join(ROOT, "include"), "-I", _cuda_include(),
                                                 os.path.join(ROOT, "tests", "native", "layout_check.cpp"), "-o", so])
    L = C.CDLL(so)
    L.ly_wavefront_bytes.restype = C.c_uint64
    L.ly_wavefront_bytes.argtypes = [C.c_uint64, C.c_int]
    return L


def test_wavefront_state(ly):
    """13 float4 and one uint4 of state a path, and 14 queues of path ids; 16
    counters a bounce, in a block of whole 256 bytes."""
    paths = 1 << 20
    assert ly.ly_wavefront_bytes(paths, 34) <= paths * (14 * 16 + 14 * 4) + 34 * 64 + 255


@pytest.mark.gpu
def test_adjoint_records_kept_by_a_context():
    """The records of a deep frame (4 GiB a batch) are given back when the call ends:
    a context keeps 2 GiB at most, and the calls that follow give the same."""
    import numpy as np
    import torch
    with cg.Context(device=0) as ctx:
        sid = ctx.upload(scenes.diff_scene(width=1024, height=1024, spp=4, max_depth=200, n_spheres=6, subdivision=1,
                                           tex_size=8, n_conductors=2, n_lights=2, seed=5))
        W = np.full((1024, 1024, 3), 1e-3, np.float32)
        ctx.adjoint_forward(sid, 1, 3)  # the path state and the gradient buffers
        before = torch.cuda.mem_get_info()[0]
        first = ctx.adjoint_backward(sid, 1, 3, W)
        assert before - torch.cuda.mem_get_info()[0] < (2 << 30) + (64 << 20)
        for a, b in zip(first, ctx.adjoint_backward(sid, 1, 3, W)):
            np.testing.assert_allclose(a, b, rtol=1e-9, atol=1e-12 * np.abs(a).max())


@pytest.mark.gpu
def test_reordering_sorts_one_ray_a_path(gpu_ctx):
    """Keys and values twice, four bytes each, and less than a byte of counts."""
    import torch
    sid = gpu_ctx.upload(scenes.cornell_box(64, 64, 1, 4))
    base = gpu_ctx.tuning()
    paths = 1 << 23
    free = []
    try:
        for reorder in (0, 4):
            gpu_ctx.set_tuning(64, 64, paths, reorder=reorder)
            gpu_ctx.render([sid], 0, 1, seed=1)
            free.append(torch.cuda.mem_get_info()[0])
    finally:
        gpu_ctx.set_tuning_dict(base)
        gpu_ctx.release(sid)
    assert 16 * paths <= free[0] - free[1] < 17 * paths + (16 << 20)
