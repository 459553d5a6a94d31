"""Ray queries that reach behind their origin (negative t_min, t_max): the walls of
a box have boxes without thickness, and a bound that is scaled rather than
widened shrinks for a negative distance."""
import ctypes as C

import numpy as np
import pytest

from cadise_gb300 import abi, scenes
from golden_scenes import specs
from test_tie_hit import tc  # noqa: F401

NAMES = ["cornell", "coplanar", "features", "field"]


def behind(n, lo, hi, seed):
    """Rays in [lo, hi] of which most have a negative t_min, some a negative t_max."""
    rng = np.random.default_rng(seed)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = lo + (hi - lo) * rng.random((n, 3))
    d = rng.normal(0, 1, (n, 3))
    d[: n // 8] = np.eye(3)[rng.integers(0, 3, n // 8)] * np.where(rng.random(n // 8) < 0.5, 1, -1)[:, None]
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    size = np.linalg.norm(hi - lo)
    rays[:, 3] = -rng.uniform(0, 4, n) * size
    rays[:, 7] = 3.4e38
    rays[n // 2:, 7] = rng.uniform(-1, 0.5, n - n // 2) * size
    rays[: n // 4, 3] = -1e4 * size
    return rays


def every_record(tc, spec, rays):  # noqa: F811
    """Per ray the smallest distance of all records of the scene, then the two
    traversals' on the CPU; the any-hit traversal's answer; the tie window."""
    flat = abi.flatten(spec)
    err = C.create_string_buffer(512)
    scene = tc.tc_create(C.addressof(flat.desc), err, 512)
    assert scene, err.value
    n = len(rays)
    t, hits, window = np.zeros((n, 3), np.float32), np.zeros(n, np.int32), np.zeros(n, np.float32)
    tc.tc_closest.argtypes = [C.c_void_p, C.c_void_p, C.c_uint32] + [C.c_void_p] * 3
    tc.tc_closest(scene, rays.ctypes.data, n, t.ctypes.data, hits.ctypes.data, window.ctypes.data)
    tc.tc_destroy(scene)
    found = t[:, 0] < 3e38
    assert found.mean() > 0.2 and (t[found, 0] < 0).mean() > 0.2
    return t, hits != 0, window, found


def rays_in(spec, n):
    points = np.concatenate([p.positions.reshape(-1, 3) if isinstance(p, scenes.TriangleMesh) else
                             np.array([p.v1, p.v2, p.v3]) for p in spec.primitives])
    return behind(n, *np.percentile(points, [10, 90], axis=0), 4)


@pytest.mark.parametrize("name", NAMES)
def test_traversals_find_hits_behind_the_origin(tc, name):  # noqa: F811
    rays = rays_in(specs()[name], 4000)
    t, hits, window, found = every_record(tc, specs()[name], rays)
    assert np.array_equal(hits, found)
    for k in (1, 2):
        assert np.array_equal(t[:, k] < 3e38, found)
        # within the tie window the reference's rule may order another hit first
        assert np.all(np.abs(t[found, k] - t[found, 0]) <= 2 * window[found])


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_queries_find_hits_behind_the_origin(gpu_ctx, tc, name):  # noqa: F811
    """Few rays (one a thread) and, the same ones over and over, many (the
    persistent pass)."""
    spec = specs()[name]
    rays = rays_in(spec, 4000)
    t, _, window, found = every_record(tc, spec, rays)
    sid = gpu_ctx.upload(spec)
    for copies in (1, 34):
        many = np.tile(rays, (copies, 1))
        prim, got, _, _ = gpu_ctx.trace_closest(sid, many)
        prim, got = prim.reshape(copies, -1), got.reshape(copies, -1)
        assert np.array_equal(prim >= 0, np.broadcast_to(found, prim.shape))
        # the answer is the reference's distance, which the window is there to bound
        assert np.all(np.abs(got - t[:, 0])[:, found] <= 2 * window[found])
        assert np.array_equal(gpu_ctx.trace_any(sid, many).reshape(copies, -1) != 0, np.broadcast_to(found, prim.shape))
    gpu_ctx.release(sid)
