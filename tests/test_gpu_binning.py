"""The fused rebin's refs through cells of 8x8 tiles (entries per (splat,
cell), sorted by cell, expanded in place) against the six reference stages:
keys, values and tile ranges bit for bit, at the edges of its tiling - grids a
tile over or under whole cells, cells of no entry, of one, of several chunks of
1024, chunks of more refs than one window of 10,240 holds, splats over the whole
grid, grids of more than 256 tiles per axis, cell counts around a digit.  The
cells serve scenes of 300,000 splats or more, so each scene is filled up to that
with splats behind the camera."""
import numpy as np
import pytest

from gs3d import GaussianSplatRenderer, Scene, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer(built_lib):
    r = GaussianSplatRenderer(Scene())
    r.init()
    yield r
    r.destroy()


TOTAL = 300_100


def cloud(n, seed, spread, scale):
    rng = np.random.default_rng(seed)
    xyz = np.tile(np.float64([0.0, 0.0, 50.0]), (TOTAL, 1))
    at = np.sort(rng.choice(TOTAL, n, replace=False))
    xyz[at] = rng.normal(0, spread, (n, 3))
    return scenes.activate(xyz, rng.normal(0, 0.5, (TOTAL, 3)), rng.normal(0, 1.5, TOTAL),
                           rng.normal(np.log(scale), 0.7, (TOTAL, 3)),
                           rng.standard_normal((TOTAL, 4)))


def refs(r, data, tile, w, h, stagewise):
    u = scenes.camera_at((0.3, 0.2, 6.0), w, h).getUniformData(w, h)
    r.setStagewise(stagewise)
    r.rebin(data.splatCount, -(-w // tile[0]), -(-h // tile[1]), w, h, u)
    r.setStagewise(False)
    R = r.refCount()
    return (R, r.readBuffer("sort_keys_a", R), r.readBuffer("sort_values_a", R),
            r.readBuffer("tile_offsets"), r.readImage().view(np.uint16).copy())


@pytest.mark.parametrize("n,spread,scale,tile,w,h", [
    (1, 0.0, 5.0, (8, 8), 264, 72),        # one splat over 33 x 9 tiles: every cell one entry
    (1, 0.0, 0.001, (8, 8), 512, 128),     # one ref: all other cells empty
    (900, 1.0, 0.02, (8, 8), 200, 136),    # 25 x 17 tiles: ragged cells
    (5000, 0.02, 0.01, (16, 16), 640, 480),  # one cell holds nearly all: several chunks
    (3000, 1.0, 1.5, (8, 8), 320, 256),    # whole-cell rectangles: many windows a chunk
    (200, 1.5, 0.3, (4, 4), 1200, 100),    # 300 tiles across: no one-word rectangles
    (4000, 1.5, 0.05, (8, 8), 1024, 1024),  # 256 cells: one digit exactly
    (4000, 1.5, 0.05, (8, 8), 1032, 1024),  # 272 cells: two digits
    (4000, 1.5, 0.05, (1, 1), 150, 90),    # 13,500 tiles of one pixel
    (4000, 60.0, 0.05, (8, 8), 640, 480),  # mostly culled
])
def test_refs_equal_the_reference_stages(renderer, n, spread, scale, tile, w, h):
    r = renderer
    data = cloud(n, n, spread, scale)
    r.setSplatData(data)
    r.setTileSize(*tile)
    want = refs(r, data, tile, w, h, True)
    got = refs(r, data, tile, w, h, False)
    assert want[0] > 0 and want[3].size > 257
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    r.setTileSize(16, 16)


@pytest.mark.parametrize("scale", [0.1, 0.2, 0.3, 0.45, 0.7])
def test_chunks_around_one_window(renderer, scale):
    """Chunks of 4 to 40 refs an entry: placed a tile a lane up to one window
    of refs, an entry a lane beyond it."""
    r = renderer
    data = cloud(6000, 77, 1.0, scale)
    r.setSplatData(data)
    r.setTileSize(8, 8)
    want = refs(r, data, (8, 8), 400, 300, True)
    got = refs(r, data, (8, 8), 400, 300, False)
    assert want[0] > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    r.setTileSize(16, 16)


def test_overflow_grows_and_repeats(renderer):
    """More refs than the key buffers hold (16 per splat at first): nothing is
    written, the count is reported exactly and the repeated rebin is whole."""
    r = GaussianSplatRenderer(Scene())
    r.init()
    try:
        data = cloud(20_000, 5, 0.5, 2.0)
        r.setSplatData(data)
        w, h = 640, 480
        u = scenes.camera_at((0.3, 0.2, 6.0), w, h).getUniformData(w, h)
        r.rebin(data.splatCount, 40, 30, w, h, u, check=False)
        with pytest.raises(Exception) as e:
            r.synchronize()
        assert "exceeded the key capacity" in str(e.value)
        want = refs(r, data, (16, 16), w, h, True)
        got = refs(r, data, (16, 16), w, h, False)
        assert want[0] > 16 * TOTAL
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
    finally:
        r.destroy()
