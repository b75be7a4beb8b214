"""Full-size images against the raster that shades pixel by pixel without a cull
(tiles of 15x15 pixels; an image does not depend on the tile grid), bit for bit:
regions of 2x2 blocks, blocks handed on, half blocks, and degenerate splats."""
import numpy as np
import pytest

from gs3d import GaussianSplatRenderer, Scene, _lib, scenes

from test_gpu_robustness import _degenerate_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer(built_lib):
    r = GaussianSplatRenderer(Scene())
    r.init()
    yield r
    r.destroy()


def image(r, data, tile, u, w, h, schedule=_lib.SCHEDULE_ROW_MAJOR):
    r.setTuning(tile, 8, 0)
    r.setSchedule(schedule)
    r.rebin(data.splatCount, -(-w // tile[0]), -(-h // tile[1]), w, h, u)
    r.setSchedule(_lib.SCHEDULE_ROW_MAJOR)
    return r.readImage().view(np.uint16).copy()


@pytest.mark.parametrize("w,h", [(640, 360), (333, 217)])
def test_degenerate_splats(renderer, w, h):
    data = _degenerate_scene()
    u = scenes.small_camera(w, h).getUniformData(w, h)
    renderer.setSplatData(data)
    want = image(renderer, data, (15, 15), u, w, h)
    assert want.any()
    for tile in [(16, 16), (32, 32), (64, 32), (12, 8), (24, 20)]:
        assert np.array_equal(image(renderer, data, tile, u, w, h), want), tile


@pytest.mark.slow
def test_a_full_capture(renderer):
    w, h = 1920, 1080
    data = scenes.scene_clusters(3_000_000, seed=1, sh_degree=3)
    u = scenes.camera_at(scenes.orbit_eyes(1, radius=12.0, seed=2)[0], w, h).getUniformData(w, h)
    renderer.setSplatData(data)
    want = image(renderer, data, (15, 15), u, w, h)
    for tile in [(16, 16), (64, 32)]:
        assert np.array_equal(image(renderer, data, tile, u, w, h), want), tile


@pytest.mark.slow
def test_long_lists_handed_on_and_split(renderer):
    w, h = 1920, 1080
    data = scenes.scene_opacity_mix(500_000, 150_000, seed=3)
    u = scenes.camera_at(scenes.random_eyes(1, 9.0, 12.0, seed=9)[0], w, h).getUniformData(w, h)
    renderer.setSplatData(data)
    want = image(renderer, data, (15, 15), u, w, h)
    sent = 0
    for _ in range(3):
        assert np.array_equal(image(renderer, data, (16, 16), u, w, h), want)
        sent += int(renderer.readBuffer("raster_pool")[0])
    assert sent > 0
    got = image(renderer, data, (16, 16), u, w, h, _lib.SCHEDULE_KEY_COUNT)
    assert np.array_equal(got, want) and renderer.getScheduleStatus()["split_tiles"] > 0
