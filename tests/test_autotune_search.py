"""The autotuner's search where the tuning leaves the traversal variant open: what
that stands for is decided by the launches, not by the number, and one ray per
thread can be asked for whatever the library would choose."""
import ctypes as C
import json
import os
import subprocess

import numpy as np
import pytest

from cadise_gb300 import abi, scenes

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
TRAVERSAL, BLOCK_TRACE, BLOCK_SHADE, MAX_PATHS, REFILL_CLOSEST, REFILL_ANY = range(6)
OPEN, REPLACE, PERSISTENT_CLOSEST, PERSISTENT, PER_RAY = range(5)


@pytest.fixture(scope="module")
def tn(tmp_path_factory):
    from cadise_gb300.native_build import CXX_FLAGS, _cuda_include
    so = str(tmp_path_factory.mktemp("tn") / "tune_check.so")
    subprocess.check_call(["g++"] + CXX_FLAGS + ["-shared", "-I", os.path.join(ROOT, "include"), "-I", _cuda_include(),
                                                 os.path.join(ROOT, "tests", "native", "tune_check.cpp"), "-o", so])
    return C.CDLL(so)


def tuning(**kw):
    return abi.cgpu_tuning(**dict({"block_trace": 64, "block_shade": 128, "max_paths": 1 << 20}, **kw))


def test_variants(tn):
    assert [tn.tn_kernels(t, 0) for t in range(5)] == [0, 1, 2, 3, 0]
    assert [tn.tn_kernels(t, 1) for t in range(5)] == [3, 1, 2, 3, 0]


@pytest.mark.parametrize("kernels", [0, 1, 2, 3])
@pytest.mark.parametrize("open_", [False, True])
def test_search_goes_by_the_launches(tn, kernels, open_):
    """`best` took `kernels`, by its own number or with the choice left open."""
    best = tuning(traversal=OPEN if open_ else kernels or PER_RAY)

    def skips(which, **kw):
        t = tuning(**dict({"traversal": best.traversal}, **kw))
        return bool(tn.tn_skips(which, C.byref(t), C.byref(best), kernels, kernels))

    assert [skips(TRAVERSAL, traversal=t) for t in (REPLACE, PERSISTENT_CLOSEST, PERSISTENT, PER_RAY)] == [
        kernels == 1, kernels == 2, kernels == 3, kernels == 0]
    assert skips(BLOCK_TRACE, block_trace=64) and not skips(BLOCK_TRACE, block_trace=128)
    assert skips(BLOCK_SHADE, block_shade=128) and not skips(BLOCK_SHADE, block_shade=64)
    assert skips(MAX_PATHS, max_paths=1 << 20) and not skips(MAX_PATHS, max_paths=1 << 22)
    for v in (8, 16, 28, 32):
        assert skips(REFILL_CLOSEST, refill_closest=v) == (kernels < 2)
        assert skips(REFILL_ANY, refill_any=v) == (kernels < 3)
    assert skips(REFILL_CLOSEST, refill_closest=24) and skips(REFILL_ANY, refill_any=24)  # the default


@pytest.mark.gpu
def test_one_ray_per_thread_on_a_large_batch(gpu_ctx):
    """A frame that the open choice gives to the persistent passes (they leave
    rays to the tie kernel) runs one ray per thread where that is asked for."""
    sid = gpu_ctx.upload(scenes.icosphere_field(n_spheres=12, subdivision=2, n_lights=2, seed=3, width=640, height=420,
                                                spp=2, max_depth=4, box=30.0, radius_range=(2.0, 5.0)))
    base = gpu_ctx.tuning()
    films, ties = [], []
    try:
        for traversal in (OPEN, PER_RAY):
            gpu_ctx.set_tuning(64, 128, traversal=traversal)
            gpu_ctx.film_clear(sid)
            gpu_ctx.render([sid], 0, 2, seed=3)
            films.append(gpu_ctx.film_read(sid))
            gpu_ctx.set_profiling(True)
            gpu_ctx.render([sid], 0, 2, seed=3)
            ties.append(gpu_ctx.kernel_times()["ties"][1])
            gpu_ctx.set_profiling(False)
    finally:
        gpu_ctx.set_profiling(False)
        gpu_ctx.set_tuning_dict(base)
        gpu_ctx.release(sid)
    assert ties[0] > 0 and ties[1] == 0
    for x, y in zip(*films):
        assert np.array_equal(x, y)


@pytest.mark.gpu
def test_results_of_an_older_search_are_not_reused(gpu_ctx, tmp_path):
    """Traversal 0 in them stood for other kernels: their lines carry no mark of
    the search."""
    sid = gpu_ctx.upload(scenes.cornell_box(32, 32, 1, 4))
    base = gpu_ctx.tuning()
    cache = tmp_path / "tune.jsonl"
    try:
        gpu_ctx.autotune([sid], samples=1, cache_path=str(cache))
        line = json.loads(cache.read_text())
        assert line["key"].endswith("|search2")
        line["key"] = line["key"][:-len("|search2")]
        line["block_trace"] = 512
        cache.write_text(json.dumps(line) + "\n")
        assert gpu_ctx.autotune([sid], samples=1, cache_path=str(cache))["block_trace"] != 512
        assert len(cache.read_text().splitlines()) == 2
    finally:
        gpu_ctx.set_tuning_dict(base)
        gpu_ctx.release(sid)
