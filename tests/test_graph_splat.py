"""A captured graph is replayed for frames of any size: one that was captured on
a tiny frame accumulates the film of a large one as fast as one captured on the
large frame itself."""
import time

import numpy as np
import pytest

import cadise_gb300 as cg
from cadise_gb300 import scenes

SPP = 16


def frame(ctx, sid, spp):
    ctx.film_clear(sid)
    ctx.synchronize()
    t = time.perf_counter()
    ctx.render([sid], 0, spp, seed=3)
    return time.perf_counter() - t


@pytest.mark.gpu
def test_graph_of_a_tiny_frame_serves_a_large_one():
    """The film splat of 1280 x 720 pixels and 16 samples takes 0.3 ms of the
    frame's 14; by as many threads as the tiny frame has pixels it took 47."""
    best, films = [], []
    for tiny_first in (False, True):
        with cg.Context(device=0) as ctx:
            large = ctx.upload(scenes.cornell_box(1280, 720, SPP, 4))
            tiny = ctx.upload(scenes.cornell_box(24, 20, 1, 4))
            if tiny_first:
                frame(ctx, tiny, 1)
            best.append(min(frame(ctx, large, SPP) for _ in range(6)))
            films.append(ctx.film_read(large))
    assert best[1] < 1.5 * best[0]
    for x, y in zip(*films):
        assert np.array_equal(x, y)
