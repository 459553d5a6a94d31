"""The three ray passes of a bounce in one launch (per-ray traversal) against
the same passes launched one by one (per-kernel timing on) and the megakernel."""
import numpy as np
import pytest

from cadise_gb300 import CGPU_MODE_MEGAKERNEL, CGPU_MODE_WAVEFRONT, abi, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("make", [scenes.cornell_box, scenes.sphere_box])
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 1), (31, 1, 2, 2), (33, 31, 3, 5), (320, 200, 2, 6)])
def test_one_launch_matches_separate_passes(gpu_ctx, make, w, h, spp, depth):
    sid = gpu_ctx.upload(abi.flatten(make(w, h, spp, depth)))
    films = []
    try:
        for mode, separate in ((CGPU_MODE_WAVEFRONT, False), (CGPU_MODE_WAVEFRONT, True), (CGPU_MODE_MEGAKERNEL, False)):
            gpu_ctx.set_profiling(separate)
            gpu_ctx.film_clear(sid)
            gpu_ctx.render([sid], 0, spp, seed=4, mode=mode)
            films.append(gpu_ctx.film_read(sid))
        gpu_ctx.set_profiling(False)
        gpu_ctx.film_clear(sid)
        gpu_ctx.render_noalloc(sid, 0, spp, seed=4)
        films.append(gpu_ctx.film_read(sid))
    finally:
        gpu_ctx.set_profiling(False)
        gpu_ctx.release(sid)
    assert films[0][2].sum() > 0
    for f in films[1:]:
        for x, y in zip(films[0], f):
            np.testing.assert_allclose(x, y, rtol=1e-14, atol=0)
