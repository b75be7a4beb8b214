"""The raster on projected records written as they are: conics that are not
positive definite or not finite, means and radii that are not finite, opacities
around every bound.  A splat may be skipped for a block of pixels only where no
pixel of it passes the per-pixel tests, which a NaN alpha does (as 0.99).  Tiles
of 15x15 pixels are shaded pixel by pixel, without a cull, and an image does not
depend on the tile grid: every other shape has to give that image bit for bit."""
import numpy as np
import pytest

from gs3d import GaussianSplatRenderer, Scene, scenes
from gs3d.renderer import PROJ_DTYPE

pytestmark = pytest.mark.gpu

N = 150_000  # sizes the key buffers; the records used are the first few
LISTED = 96  # splats in every tile's list


@pytest.fixture(scope="module")
def renderer(built_lib):
    r = GaussianSplatRenderer(Scene())
    r.init()
    r.setSplatData(scenes.scene_small(N, seed=1))
    yield r
    r.destroy()


def records(rng, w, h, conic, opacity, radius, mean):
    p = np.zeros(N, PROJ_DTYPE)
    m = slice(0, LISTED)
    p["mean_px"][m] = rng.uniform(-20, [w + 20, h + 20], (LISTED, 2))
    p["depth"][m] = -np.arange(1, LISTED + 1)
    p["radius_px"][m] = rng.choice(radius, LISTED)
    p["conic"][m] = conic(rng, p["radius_px"][m][:, None])
    p["opacity"][m] = rng.choice(opacity, LISTED)
    p["color"][m] = rng.random((LISTED, 3))
    p["valid"][m] = 1
    if mean is not None:  # one in three
        p["mean_px"][0:LISTED:3, rng.integers(2)] = mean
    return p


def image(r, tile, w, h, p, split=False):
    r.setTuning(tile, 8, 0)
    r.setCamera(scenes.small_camera(w, h).getUniformData(w, h), w, h)
    tiles = (-(-w // tile[0])) * (-(-h // tile[1]))
    r.writeBuffer("projected_splats", p)
    r.writeBuffer("tile_offsets", np.arange(tiles + 1, dtype=np.uint32) * LISTED)
    r.writeBuffer("sort_values_a", np.tile(np.arange(LISTED, dtype=np.uint32), tiles))
    r.setSplitAllTiles(split)
    try:
        r.rasterizeTiles()
        r.synchronize()
    finally:
        r.setSplitAllTiles(False)
    return r.readImage().view(np.uint16).copy()


def around(sign_a, sign_c, mix):
    """Conics of terms about 4.5 / radius^2 (the edge of a 3-sigma circle) and
    `mix` times as large a mixed term."""
    def f(rng, r):
        s = 4.5 / (r * r) * rng.uniform(0.3, 1.5, (LISTED, 3))
        return s * np.float32([sign_a, mix, sign_c]) * rng.choice([-1, 1], (LISTED, 3)) ** [0, 1, 0]
    return f


def steep(rng, r):
    """Terms of some hundreds at the edge: exp underflows inside the circle."""
    return 80 * around(1, 1, 0.15)(rng, r)


def holed(value):
    """Positive definite ones, one entry of every other splat replaced."""
    def f(rng, r):
        c = around(1, 1, 0.15)(rng, r)
        i = np.arange(0, LISTED, 2)
        c[i, rng.integers(0, 3, len(i))] = value
        return c
    return f


FAINT = [0.0005, 0.0039, 1 / 255, 0.00393, 0.5]
STRONG = [0.3, 0.98, 0.98985, 0.98995, 0.9999, 1.0]
RADII = [2, 6, 20, 60]
ODD = [0.2, np.nan, np.inf, -np.inf, -1.0, 3.0, 1e30]
CASES = {
    "positive definite": (around(1, 1, 0.15), FAINT + STRONG, RADII, None),
    "nan conic": (holed(np.nan), FAINT + STRONG, RADII, None),
    "infinite conic": (holed(np.inf), FAINT + STRONG, RADII, None),
    "huge conic": (holed(3e38), FAINT + STRONG, RADII, None),
    "zero conic": (holed(0.0), FAINT + STRONG, RADII, None),
    "negative definite": (around(-1, -1, 0.2), FAINT + STRONG, RADII, None),
    "one diagonal negative": (around(-1, 1, 0.2), FAINT + STRONG, RADII, None),
    "indefinite": (around(1, 1, 6.0), FAINT + STRONG, RADII, None),
    "odd opacities": (around(1, 1, 0.15), ODD, RADII, None),
    "odd opacities, steep": (steep, ODD, RADII, None),
    "nan mean": (around(1, 1, 0.15), FAINT + STRONG, RADII, np.nan),
    "infinite mean": (around(1, 1, 0.15), FAINT + STRONG, RADII, np.inf),
    "odd radii": (around(1, 1, 0.15), FAINT + STRONG, [2, 60, np.nan, np.inf, 1e20, 0.0], None),
}


# 323x197: single blocks of 8x8; 1920x1080: regions of 2x2 blocks
@pytest.mark.parametrize("w,h", [(323, 197), (1920, 1080)])
@pytest.mark.parametrize("case", CASES)
def test_every_tile_shape_gives_the_unculled_image(renderer, case, w, h):
    conic, opacity, radius, mean = CASES[case]
    rng = np.random.default_rng(list(CASES).index(case))
    with np.errstate(all="ignore"):
        p = records(rng, w, h, conic, opacity, radius, mean)
    want = image(renderer, (15, 15), w, h, p)
    assert want.any() or case == "negative definite"  # its powers are all positive
    for tile in [(16, 16), (32, 32), (12, 8)]:
        for split in (False, True):
            got = image(renderer, tile, w, h, p, split)
            assert np.array_equal(got, want), (tile, split, int((got != want).any(-1).sum()))


@pytest.mark.parametrize("case", ["negative definite", "one diagonal negative", "indefinite"])
def test_forms_that_are_not_positive_match_the_oracle(renderer, oracle, case):
    """A positive power skips the splat there, as in the reference."""
    w, h, tile = 323, 197, (16, 16)
    conic, opacity, radius, _ = CASES[case]
    p = records(np.random.default_rng(50), w, h, conic, opacity, radius, None)
    got = image(renderer, tile, w, h, p).view(np.float16).astype(np.float32)
    tiles = (-(-w // tile[0])) * (-(-h // tile[1]))
    want = oracle.rasterize(w, h, *tile, p, np.arange(tiles + 1, dtype=np.uint32) * LISTED,
                            np.tile(np.arange(LISTED, dtype=np.uint32), tiles))
    want = want[0] if isinstance(want, tuple) else want
    assert np.abs(got - want).max() <= 2.0 / 255.0
