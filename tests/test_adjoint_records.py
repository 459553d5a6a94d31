"""The device side of the adjoint calls: the image of cgpu_adjoint_forward
against the mean of the film it is worked out from."""
import numpy as np
import pytest

from cadise_gb300 import scenes

pytestmark = pytest.mark.gpu


def small_scene(width, height, max_depth=4):
    return scenes.diff_scene(width=width, height=height, spp=4, max_depth=max_depth, n_spheres=6, subdivision=1,
                             tex_size=8, n_conductors=2, n_lights=2, seed=5)


@pytest.mark.parametrize("width,height", [(1, 1), (37, 23), (256, 1), (700, 501)])
def test_forward_image_is_the_film_mean(gpu_ctx, width, height):
    """Bit for bit: one FP64 division, rounded once."""
    sid = gpu_ctx.upload(small_scene(width, height))
    try:
        img = gpu_ctx.adjoint_forward(sid, 3, 9)
        s, _, n = gpu_ctx.film_read(sid)
        mean = np.where(n[..., None] > 0, s / np.maximum(n, 1.0)[..., None], 0.0).astype(np.float32)
        np.testing.assert_array_equal(img.reshape(mean.shape), mean)
    finally:
        gpu_ctx.release(sid)


@pytest.mark.parametrize("width,height,max_depth,spp,batches", [
    (1, 1, 1, 1, 1), (33, 31, 1, 5, 1), (127, 95, 2, 3, 1), (64, 48, 9, 16, 1),
    (1024, 1024, 200, 2, 4),  # the records of one sample do not fit a batch: each in two parts
])
def test_replay_from_records_matches_the_retracing_schedule(gpu_ctx, width, height, max_depth, spp, batches):
    """The wavefront adjoint replays from recorded hits and visibilities, the
    megakernel one traces every ray again: the same FP32 terms, so that the
    gradients agree up to the order of the FP64 sums."""
    from cadise_gb300 import CGPU_MODE_MEGAKERNEL, CGPU_MODE_WAVEFRONT
    sid = gpu_ctx.upload(small_scene(width, height, max_depth))
    try:
        W = np.random.default_rng(7).normal(size=(height, width, 3)).astype(np.float32)
        gpu_ctx.set_adjoint_mode(CGPU_MODE_MEGAKERNEL)
        ref = gpu_ctx.adjoint_backward(sid, spp, 13, W)
        gpu_ctx.set_adjoint_mode(CGPU_MODE_WAVEFRONT)
        got = gpu_ctx.adjoint_backward(sid, spp, 13, W)
        assert gpu_ctx.stats().batches == batches
        for a, b in zip(got, ref):
            scale = np.abs(b).max() if b.size else 0.0
            np.testing.assert_allclose(a, b, rtol=1e-7, atol=1e-10 * scale + 1e-30)
    finally:
        gpu_ctx.set_adjoint_mode(CGPU_MODE_WAVEFRONT)
        gpu_ctx.release(sid)
