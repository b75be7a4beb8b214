"""Elongated splats and the raster's warp cull: a warp may skip a splat only
where no pixel of its block blends it, whatever the conic's condition number.
Tiles whose area is no multiple of 32 are shaded pixel by pixel without the
cull, and an image does not depend on the tile grid, so the culled images
have to equal that one bit for bit."""
import numpy as np
import pytest

from gs3d import GaussianSplatRenderer, Scene, scenes

pytestmark = pytest.mark.gpu


def needles(n, seed, long, thin):
    """Splats of one long axis and two thin ones, any direction, some large
    enough to cross the view; opacities around the 1/255 cut-off and above."""
    rng = np.random.default_rng(seed)
    xyz = rng.normal(0.0, 2.0, (n, 3))
    scale = np.stack([rng.uniform(np.log(long) - 2.0, np.log(long), n),
                      np.full(n, np.log(thin)), rng.uniform(np.log(thin), np.log(thin) + 2, n)], 1)
    opacity = np.where(rng.random(n) < 0.2, rng.normal(-5.5, 0.1, n), rng.normal(0.5, 2.0, n))
    return scenes.activate(xyz, rng.normal(0, 0.5, (n, 3)), opacity, scale,
                           rng.standard_normal((n, 4)))


@pytest.mark.parametrize("long,thin", [(0.05, 0.01), (0.5, 1e-3), (5.0, 1e-3), (60.0, 1e-4),
                                       (2000.0, 1e-5)])
@pytest.mark.parametrize("w,h", [(320, 200), (333, 217)])
def test_culled_images_equal_the_unculled_raster(built_lib, long, thin, w, h):
    data = needles(3000, int(long * 10), long, thin)
    u = scenes.camera_at((0.4, 0.3, 7.0), w, h).getUniformData(w, h)
    r = GaussianSplatRenderer(Scene())
    r.init()
    try:
        r.setSplatData(data)
        images = {}
        for tile in [(15, 15), (16, 16), (32, 32), (64, 32), (12, 8), (24, 20)]:
            r.setTuning(tile, 8, 0)
            r.rebin(data.splatCount, -(-w // tile[0]), -(-h // tile[1]), w, h, u)
            images[tile] = r.readImage().view(np.uint16).copy()
    finally:
        r.destroy()
    want = images.pop((15, 15))
    assert want.any()
    for tile, img in images.items():
        assert np.array_equal(img, want), tile
