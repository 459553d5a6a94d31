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
