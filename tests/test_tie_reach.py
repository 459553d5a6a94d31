"""Layers within the tie window of one another, each tiled on its own, far from
the coordinate origin: where the reference's test rejects the nearest tiles (a
ray through their edge), the layer behind them is the hit.  The persistent
passes meet it whatever they visited first."""
import numpy as np
import pytest

from cadise_gb300 import CGPU_MODE_MEGAKERNEL, CGPU_MODE_WAVEFRONT, abi, scenes


def layered_floor(layers, step, tiles, offset, seed=1):
    """The Cornell box's walls moved by `offset` along every axis, its floor
    replaced by `layers` layers `step` apart (the tie window is 2^-16 of the
    offset and more)."""
    s = scenes.cornell_box(160, 120, 4, 3)
    rng = np.random.default_rng(seed)
    o = np.full(3, float(offset))
    s.primitives = [p for p in s.primitives if isinstance(p, scenes.Rectangle) and p.name != "floor"]
    for p in s.primitives:
        p.v1, p.v2, p.v3 = (tuple(np.asarray(v) + o) for v in (p.v1, p.v2, p.v3))
    s.cam_position = tuple(np.asarray(s.cam_position) + o)
    for k in range(layers):
        gx, gz = (np.concatenate([[0], np.sort(rng.uniform(0, 556, tiles - 1)), [556]]) for _ in range(2))
        u, v = np.meshgrid(gx, gz, indexing="ij")
        g = np.stack([u, np.full_like(u, step * k), v], -1)
        q = np.concatenate([np.stack([g[:-1, :-1], g[:-1, 1:], g[1:, 1:]], 2).reshape(-1, 3, 3),
                            np.stack([g[:-1, :-1], g[1:, 1:], g[1:, :-1]], 2).reshape(-1, 3, 3)])
        s.primitives.append(scenes.TriangleMesh(name="layer%d" % k, material=s.materials[k % 3].name,
                                                positions=(q + o).astype(np.float32)))
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("layers,step,tiles,offset", [(2, 0.002, 60, 3000), (4, 0.1, 200, 30000), (6, 0.02, 100, 30000),
                                                      (3, 0.4, 120, 30000)])
def test_layers_behind_the_nearest_record(gpu_ctx, layers, step, tiles, offset):
    sid = gpu_ctx.upload(abi.flatten(layered_floor(layers, step, tiles, offset)))
    base = gpu_ctx.tuning()

    def film(mode):
        gpu_ctx.film_clear(sid)
        gpu_ctx.render([sid], 0, 64, seed=6, mode=mode)
        return gpu_ctx.film_read(sid)

    try:
        ref = film(CGPU_MODE_MEGAKERNEL)
        # (traversal 0 takes the persistent passes here; the refill thresholds change which rays share a warp)
        for trav, refill in ((0, 0), (3, 0), (3, 1), (3, 32), (2, 8)):
            gpu_ctx.set_tuning(64, 64, 0, traversal=trav, refill_closest=refill)
            got = film(CGPU_MODE_WAVEFRONT)
            assert np.array_equal(got[0], ref[0]), (trav, refill, int((got[0] != ref[0]).any(-1).sum()))
    finally:
        gpu_ctx.set_tuning_dict(base)
        gpu_ctx.release(sid)
