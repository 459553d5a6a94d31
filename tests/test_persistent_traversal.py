"""The persistent traversal passes (persist.cuh): their triangle test against
tri_test to the bit, on the CPU; on the GPU their films against the
megakernel's, bit for bit, on trees whose traversal overflows the shared rows
of the stack, on queues smaller than a warp and at the ends of the refill
thresholds."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cadise_gb300 import CGPU_MODE_MEGAKERNEL, CGPU_MODE_WAVEFRONT, abi, scenes

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


@pytest.fixture(scope="module")
def pc(tmp_path_factory):
    from cadise_gb300.native_build import CXX_FLAGS, _cuda_include
    so = str(tmp_path_factory.mktemp("pc") / "persist_check.so")
    subprocess.check_call(["g++"] + CXX_FLAGS + ["-shared", "-I", os.path.join(ROOT, "include"), "-I", _cuda_include(),
                                                 os.path.join(ROOT, "tests", "native", "persist_check.cpp"), "-o", so])
    L = C.CDLL(so)
    L.pc_tri.argtypes = [C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p, C.c_void_p]
    return L


@pytest.mark.parametrize("case", ["random", "edges", "axis"])
def test_rotated_triangle_test_is_tri_test(pc, case):
    rng = np.random.default_rng(5)
    n = 200_000
    tris = rng.normal(0, 1, (n, 3, 3)).astype(np.float32)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.normal(0, 2, (n, 3))
    w = rng.dirichlet([1, 1, 1], n)
    if case == "edges":  # through vertices and edge points (zero edge functions, the 64-bit path)
        w = np.eye(3)[rng.integers(0, 3, n)]
        w[::2] = 0.5 * (w[::2] + np.eye(3)[rng.integers(0, 3, len(w[::2]))])
        tris = np.round(tris * 4) / 4
        rays[:, :3] = np.round(rays[:, :3] * 4) / 4
    target = (tris * w[:, :, None]).sum(1)
    d = target - rays[:, :3]
    d[::3] = rng.normal(0, 1, (len(d[::3]), 3))
    if case == "axis":  # one or two zero components, of either sign
        d[np.arange(n), rng.integers(0, 3, n)] = 0.0
        d[::2][np.arange(len(d[::2])), rng.integers(0, 3, len(d[::2]))] = -0.0
        d[np.all(d == 0, axis=1)] = (0, 0, -1)
    norm = np.linalg.norm(d, axis=1, keepdims=True)
    d = np.where(norm > 0, d / np.maximum(norm, 1e-30), [[1.0, 0, 0]])
    rays[:, 3] = 1e-3
    rays[:, 4:7] = d
    rays[:, 7] = np.where(rng.random(n) < 0.5, np.float32(3.4e38), rng.uniform(0, 5, n).astype(np.float32))
    rays, tris = np.ascontiguousarray(rays, np.float32), np.ascontiguousarray(tris.reshape(n, 9), np.float32)
    hit = np.zeros((n, 2), np.int32)
    t = np.zeros((n, 2), np.float32)
    pc.pc_tri(rays.ctypes.data, tris.ctypes.data, n, hit.ctypes.data, t.ctypes.data)
    assert np.array_equal(hit[:, 0], hit[:, 1])
    assert np.array_equal(t[:, 0], t[:, 1])
    assert hit[:, 0].sum() > n // 20


def shells(n, spheres=False):
    """A box of n large overlapping triangles in random planes (every ray
    crosses most boxes, so its stack runs far beyond 16 entries)."""
    s = scenes.sphere_box(24, 20, 4, 4) if spheres else scenes.cornell_box(24, 20, 4, 4)
    rng = np.random.default_rng(n)
    c = np.array([280.0, 270.0, -300.0 if spheres else 280.0])
    tri = c + rng.normal(0, 1, (n, 3, 3)) * rng.uniform(20, 260, (n, 1, 1))
    s.primitives.append(scenes.TriangleMesh(name="shells", material=s.materials[1].name, positions=tri.astype(np.float32)))
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("n,spheres", [(1, False), (40, True), (700, False), (6000, False), (6000, True)])
def test_deep_stacks_match_the_megakernel(gpu_ctx, n, spheres):
    sid = gpu_ctx.upload(abi.flatten(shells(n, spheres)))
    base = gpu_ctx.tuning()

    def film(mode):
        gpu_ctx.film_clear(sid)
        gpu_ctx.render([sid], 0, 4, seed=3, mode=mode)
        return gpu_ctx.film_read(sid)

    ref = film(CGPU_MODE_MEGAKERNEL)
    try:
        for trav, block, rc, ra in ((3, 64, 0, 0), (3, 32, 1, 1), (3, 256, 32, 32), (2, 128, 17, 0)):
            gpu_ctx.set_tuning(block, 128, 0, traversal=trav, refill_closest=rc, refill_any=ra)
            for x, y in zip(ref, film(CGPU_MODE_WAVEFRONT)):
                assert np.array_equal(x, y), (trav, block, rc, ra)
    finally:
        gpu_ctx.set_tuning_dict(base)
        gpu_ctx.release(sid)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (3, 5), (31, 1), (33, 31)])
def test_tiny_queues_match_the_megakernel(gpu_ctx, w, h):
    s = scenes.cornell_box(w, h, 1, 6)
    sid = gpu_ctx.upload(abi.flatten(s))
    base = gpu_ctx.tuning()
    films = []
    try:
        gpu_ctx.set_tuning(64, 64, 0, traversal=3)
        for mode in (CGPU_MODE_MEGAKERNEL, CGPU_MODE_WAVEFRONT):
            gpu_ctx.film_clear(sid)
            gpu_ctx.render([sid], 0, 1, seed=8, mode=mode)
            films.append(gpu_ctx.film_read(sid))
    finally:
        gpu_ctx.set_tuning_dict(base)
        gpu_ctx.release(sid)
    for x, y in zip(*films):
        assert np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["field", "features", "spheres", "coplanar", "shells"])
def test_query_batches_match_small_queries(gpu_ctx, name):
    """A batch that goes through the persistent pass gives the answers of the
    same rays asked in pieces that do not: random rays, rays with their own
    (also negative) t_min and short t_max, zero direction components,
    unnormalised directions, rays that start on a surface."""
    from golden_scenes import specs
    spec = shells(700) if name == "shells" else specs()[name]
    sid = gpu_ctx.upload(abi.flatten(spec))
    info = gpu_ctx.info(sid)
    lo, hi = np.array(info.bounds_min), np.array(info.bounds_max)
    rng = np.random.default_rng(9)
    n = (1 << 17) + 33
    size = np.linalg.norm(hi - lo)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = lo - 0.1 * (hi - lo) + 1.2 * (hi - lo) * rng.random((n, 3))
    rays[:, 4:7] = rng.normal(0, 1, (n, 3)) * rng.uniform(0.1, 10, (n, 1))
    rays[:, 3] = 1e-3
    rays[:, 7] = 3.4e38
    k = n // 8
    rays[:k, 3] = rng.uniform(-0.5, 0.5, k) * size
    rays[k:2 * k, 7] = rng.uniform(0, 0.3, k) * size
    rays[2 * k:3 * k, 4 + rng.integers(0, 3)] = 0.0
    rays[3 * k:4 * k, 4] = -0.0
    rays[3 * k:4 * k, 5] = 0.0
    prim, t, _, _ = gpu_ctx.trace_closest(sid, rays[4 * k:5 * k])
    d = rays[4 * k:5 * k, 4:7] / np.linalg.norm(rays[4 * k:5 * k, 4:7], axis=1, keepdims=True)
    rays[5 * k:6 * k, :3] = rays[4 * k:5 * k, :3] + d * t[:, None]  # (misses: their own origin)
    whole = gpu_ctx.trace_closest(sid, rays), (gpu_ctx.trace_any(sid, rays),)
    parts = [(gpu_ctx.trace_closest(sid, rays[i:i + 1000]), (gpu_ctx.trace_any(sid, rays[i:i + 1000]),))
             for i in range(0, n, 1000)]
    for q in (0, 1):
        for j in range(len(whole[q])):
            assert np.array_equal(whole[q][j], np.concatenate([p[q][j] for p in parts])), (name, q, j)
    gpu_ctx.release(sid)


@pytest.mark.gpu
@pytest.mark.parametrize("layers,step", [(2, 0.0), (3, 0.0), (3, 1e-3), (7, 5e-4)])
def test_layers_within_the_tie_window(gpu_ctx, layers, step):
    """Several primitives within the tie window (2^-16 of the scene's 560 units)
    of every hit on a tilted sheet: the nearest is traced again within its
    window.  Render against the megakernel, a large batch of queries (hits
    before and behind the origin, t_max on the sheet) against small ones."""
    s = scenes.cornell_box(48, 40, 4, 4)
    m = 24
    u, v = np.meshgrid(np.linspace(60, 500, m), np.linspace(60, 500, m), indexing="ij")
    g = np.stack([u, v, 150.0 + 0.3 * u - 0.2 * v], -1)
    quads = np.concatenate([np.stack([g[:-1, :-1], g[1:, :-1], g[1:, 1:]], 2).reshape(-1, 3, 3),
                            np.stack([g[:-1, :-1], g[1:, 1:], g[:-1, 1:]], 2).reshape(-1, 3, 3)])
    tri = np.concatenate([quads + [0, 0, step * k] for k in range(layers)]).astype(np.float32)
    s.primitives.append(scenes.TriangleMesh(name="sheet", material=s.materials[1].name, positions=tri))
    sid = gpu_ctx.upload(abi.flatten(s))
    base = gpu_ctx.tuning()
    films = []
    try:
        gpu_ctx.set_tuning(64, 64, 0, traversal=3)
        for mode in (CGPU_MODE_MEGAKERNEL, CGPU_MODE_WAVEFRONT):
            gpu_ctx.film_clear(sid)
            gpu_ctx.render([sid], 0, 4, seed=8, mode=mode)
            films.append(gpu_ctx.film_read(sid))
        for x, y in zip(*films):
            assert np.array_equal(x, y)
        n = (1 << 17) + 5
        rng = np.random.default_rng(layers)
        rays = np.zeros((n, 8), np.float32)
        rays[:, :3] = rng.uniform(50, 510, (n, 3))
        rays[:, 4:7] = rng.normal(0, 1, (n, 3))
        rays[:, 3], rays[:, 7] = 1e-3, 3.4e38
        rays[:n // 3, 3] = -1000.0
        rays[n // 3:n // 2, 7] = gpu_ctx.trace_closest(sid, rays[n // 3:n // 2])[1]
        whole = gpu_ctx.trace_closest(sid, rays)
        assert (whole[0] >= 0).mean() > 0.5 and (whole[1] < 0).any()
        parts = [gpu_ctx.trace_closest(sid, rays[i:i + 4000]) for i in range(0, n, 4000)]
        for j in range(len(whole)):
            assert np.array_equal(whole[j], np.concatenate([p[j] for p in parts])), j
    finally:
        gpu_ctx.set_tuning_dict(base)
        gpu_ctx.release(sid)
