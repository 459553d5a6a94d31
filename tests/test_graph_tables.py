"""Captured graphs and the scene tables they were captured with: once uploads
outgrow the tables, a render through a graph gives the films of direct launches,
for scenes on both sides of the growth and whichever graph was captured first."""
import numpy as np
import pytest

import cadise_gb300 as cg
from cadise_gb300 import scenes

# tables are allocated for at least this many scenes
FIRST_CAPACITY = 8


def film(ctx, sid, spp, graph):
    ctx.film_clear(sid)
    ctx.render([sid], 0, spp, seed=6, graph=graph)
    return ctx.film_read(sid)


def small(k):
    return scenes.cornell_box(24 + k, 20, 4, 4)


@pytest.mark.gpu
@pytest.mark.parametrize("between", [False, True])
def test_graphs_follow_tables_that_grow(between):
    """`between`: a render that takes the other graph (persistent passes, its own
    depth) stands between the growth and the replay."""
    with cg.Context(device=0) as ctx:
        ids = [ctx.upload(small(0))]
        large = ctx.upload(scenes.icosphere_field(n_spheres=12, subdivision=2, n_lights=2, seed=3, width=640, height=420,
                                                  spp=2, max_depth=5, box=30.0, radius_range=(2.0, 5.0)))
        film(ctx, ids[0], 3, True)  # captures, with tables of FIRST_CAPACITY scenes
        ids += [ctx.upload(small(k)) for k in range(1, FIRST_CAPACITY)]
        assert max(ids) >= FIRST_CAPACITY
        if between:
            film(ctx, large, 2, True)
        for sid in (ids[0], ids[1], ids[-1]):
            got, ref = film(ctx, sid, 3, True), film(ctx, sid, 3, False)
            assert got[2].sum() > 0
            for x, y in zip(got, ref):
                assert np.array_equal(x, y), sid
