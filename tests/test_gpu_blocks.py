"""The largest blocks that the megakernel's registers allow, with and without
counters: they launch, and give the films of small blocks."""
import numpy as np
import pytest

from cadise_gb300 import CGPU_MODE_MEGAKERNEL, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("counting", [False, True])
@pytest.mark.parametrize("block", [416, 512])
@pytest.mark.parametrize("make", [scenes.cornell_box, scenes.sphere_box])
def test_megakernel_takes_large_blocks(gpu_ctx, make, block, counting):
    sid = gpu_ctx.upload(make(48, 40, 2, 4))
    base = gpu_ctx.tuning()
    films = []
    try:
        gpu_ctx.set_counting(counting)
        for b in (64, block):
            gpu_ctx.set_tuning(b, 64)
            gpu_ctx.film_clear(sid)
            gpu_ctx.render([sid], 0, 2, seed=4, mode=CGPU_MODE_MEGAKERNEL)
            films.append(gpu_ctx.film_read(sid))
    finally:
        gpu_ctx.set_counting(False)
        gpu_ctx.set_tuning_dict(base)
        gpu_ctx.release(sid)
    assert films[0][2].sum() > 0
    for x, y in zip(*films):
        assert np.array_equal(x, y)
