"""Blocks handed on between raster warps: a few tiles at the end of the row-major
order have lists of thousands of splats, so their warps still work when the queue
has run empty, and warps that wait take over blocks of theirs.  The image and the
costs are those of half-block items, which are never handed on - also where the
waiting warps leave before a block comes, which its sender then takes back."""
import ctypes as C

import numpy as np
import pytest

from gs3d import GaussianSplatRenderer, Scene, _lib, learned, scenes
from gs3d.renderer import PROJ_DTYPE

pytestmark = pytest.mark.gpu

W, H, TX, TILES = 1920, 1080, 120, 120 * 68
HEAVY, EACH, TURNS = 40, 3000, 4  # heavy tiles, records of each, times listed
N = HEAVY * EACH + 1000


def scene():
    """Records and lists: small splats on the corners of a heavy tile's pixels, so
    that they may hit it and blend nothing, and one in twenty that blends a little."""
    rng = np.random.default_rng(4)
    heavy = TILES - 1 - 7 * np.arange(HEAVY)
    p = np.zeros(N, PROJ_DTYPE)
    p["valid"], p["depth"] = 1, -np.arange(1, N + 1)
    p["color"] = rng.random((N, 3))
    faint = rng.random(N) < 0.05
    p["radius_px"] = np.where(faint, 4, 2)
    p["conic"] = np.where(faint[:, None], [0.3, 0.05, 0.4], [60.0, 1.0, 60.0])
    p["opacity"] = np.where(faint, 0.02, 0.5)
    at = rng.integers(1, 16, (N, 2))
    for i, t in enumerate(heavy):
        p["mean_px"][i * EACH:(i + 1) * EACH] = at[i * EACH:(i + 1) * EACH] + \
            [t % TX * 16, t // TX * 16]
    light = np.arange(HEAVY * EACH, N)
    p["mean_px"][light] = rng.uniform(0, [W, H], (len(light), 2))
    p["radius_px"][light], p["opacity"][light] = 90, 0.2
    p["conic"][light] = [1e-3, 0, 1e-3]
    lists = [rng.choice(light, 24) for _ in range(TILES)]
    for i, t in enumerate(heavy):
        lists[t] = np.tile(np.arange(i * EACH, (i + 1) * EACH), TURNS)
    return p, lists


@pytest.fixture(scope="module")
def frame(built_lib):
    r = GaussianSplatRenderer(Scene())
    r.init()
    r.setSplatData(scenes.scene_small(N, seed=1))
    p, lists = scene()
    r.setTuning(16, 8, 0)
    r.setCamera(scenes.small_camera(W, H).getUniformData(W, H), W, H)
    r.writeBuffer("projected_splats", p)
    r.writeBuffer("tile_offsets", np.cumsum([0] + [len(x) for x in lists]).astype(np.uint32))
    r.writeBuffer("sort_values_a", np.concatenate(lists).astype(np.uint32))

    def shade(split=False, brief=False):
        r.setSplitAllTiles(split)
        r.setBriefWaits(brief)
        r.rasterizeTiles()
        r.synchronize()
        return (r.readImage().view(np.uint16).copy(), r.readBuffer("tile_costs"),
                r.readBuffer("raster_pool"))
    yield shade
    r.destroy()


def test_blocks_of_long_lists_are_handed_on(frame):
    image, costs, pool = frame(split=True)
    assert image.any() and (costs == EACH * TURNS).sum() == HEAVY and pool[0] == 0
    for _ in range(5):
        got, gotc, pool = frame()
        sent, places, waiting, present, expired, back = pool[:6]
        assert sent > back and places > 0 and expired == waiting == present == 0
        assert np.array_equal(got, image) and np.array_equal(gotc, costs)


def test_blocks_that_nobody_waits_for_are_taken_back(frame):
    image, costs, _ = frame(split=True)
    for _ in range(5):
        got, gotc, pool = frame(brief=True)
        assert pool[4] > 0 and pool[5] > 0  # waits that ran out, blocks taken back
        assert np.array_equal(got, image) and np.array_equal(gotc, costs)
        got, gotc, pool = frame()  # nothing is left behind for the next launch
        assert pool[0] > pool[5] and pool[4] == 0
        assert np.array_equal(got, image) and np.array_equal(gotc, costs)


def test_an_order_by_predictions_hands_on_too(built_lib):
    """A prediction may rank a long list last: batches of any size in learned order
    hand blocks on (here an untrained model's order, 11 regions a warp), and give
    the row-major order's images."""
    w, h = 1920, 1080
    data = scenes.scene_opacity_mix(300_000, 100_000, seed=3)
    eyes = scenes.random_eyes(4, 9.0, 16.0, seed=9)
    views = [(0, scenes.camera_at(e, w, h).getUniformData(w, h), w, h) for e in eyes]
    r = GaussianSplatRenderer(Scene())
    r.init()
    try:
        r.setSplatData(data)
        r.setTuning(16, 8, 0)

        def batch():
            r.rebinBatch(views)
            return ([r.readViewImage(v).view(np.uint16).copy() for v in range(4)],
                    r.readBuffer("raster_pool"))
        want, _ = batch()
        f32 = lambda *a: np.ascontiguousarray(*a, np.float32)  # noqa: E731
        p, mean, std = f32(learned.init_params(1)), f32(np.zeros(16)), f32(np.ones(16))
        r.setScheduleGate(1e9)  # the model is not trained
        r._call("gs3d_set_cost_model", *(a.ctypes.data_as(C.c_void_p) for a in (p, mean, std)))
        r.setSchedule(_lib.SCHEDULE_LEARNED)
        taken = 0
        for _ in range(3):
            got, pool = batch()
            assert r.getScheduleStatus()["active"] == _lib.SCHEDULE_LEARNED
            taken += int(pool[0]) - int(pool[5])
            for a, b in zip(got, want):
                assert np.array_equal(a, b)
        assert taken > 0
    finally:
        r.destroy()
