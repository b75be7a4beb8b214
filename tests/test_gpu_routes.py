"""Routes that a frame takes by its size, its options or what is under way beside it:
raster orders of more than 65,536 tiles, cells sorted by other digits, replays with
new cameras through cells, blocks handed on in two contexts at a time, copies of the
last frame under way while the next one starts."""
import ctypes as C
import threading

import numpy as np
import pytest

from gs3d import GaussianSplatRenderer, Scene, _lib, learned, scenes

from test_gpu_binning import cloud, refs
from test_gpu_hand_on import H, N, W, scene as long_lists

pytestmark = pytest.mark.gpu


def make():
    r = GaussianSplatRenderer(Scene())
    r.init()
    return r


@pytest.fixture
def renderer(built_lib):
    r = make()
    yield r
    r.destroy()


@pytest.mark.parametrize("w,h", [(2080, 2080), (2048, 2048), (2056, 2048)])  # 67,600, 65,536, 65,792
def test_orders_of_many_tiles(renderer, w, h):
    r = renderer
    data = scenes.scene_small(120_000, seed=8)
    u = scenes.small_camera(w, h).getUniformData(w, h)
    r.setSplatData(data)
    r.setTuning(8, 8, 0)

    def frame():
        r.rebin(data.splatCount, -(-w // 8), -(-h // 8), w, h, u)
        return r.readImage().view(np.uint16).copy(), r.readBuffer("tile_costs")
    want = frame()
    f32 = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    p, mean, std = f32(learned.init_params(1)), f32(np.zeros(16)), f32(np.ones(16))
    r.setScheduleGate(1e9)  # the model is not trained
    r._call("gs3d_set_cost_model", *(a.ctypes.data_as(C.c_void_p) for a in (p, mean, std)))
    for schedule in (_lib.SCHEDULE_KEY_COUNT, _lib.SCHEDULE_LEARNED):
        r.setSchedule(schedule)
        for split in (False, True):
            r.setSplitAllTiles(split)
            for a, b in zip(frame(), want):
                assert np.array_equal(a, b), (schedule, split)
            assert r.getScheduleStatus()["active"] == schedule


@pytest.mark.parametrize("digit", [4, 6, 8, 11])
@pytest.mark.parametrize("w,h", [(520, 264), (1032, 1024), (2400, 1800)])  # 45, 272, 1102 cells
def test_cells_sorted_by_other_digits(renderer, digit, w, h):
    r = renderer
    data = cloud(6000, digit, 1.5, 0.05)
    r.setSplatData(data)
    r.setTuning(8, digit, 0)
    want, got = (refs(r, data, (8, 8), w, h, stagewise) for stagewise in (True, False))
    assert want[0] > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_replays_with_new_cameras_through_cells(renderer):
    r = renderer
    data = scenes.scene_clusters(200_000, seed=4, sh_degree=1)
    r.setSplatData(data)
    r.setTuning(16, 8, 0)
    sets = [[(0, scenes.camera_at(e, w, h).getUniformData(w, h), w, h)
             for e, (w, h) in zip(scenes.orbit_eyes(2, radius=10.0 + k, jitter_deg=20.0, seed=k),
                                  [(960, 540), (1000, 563)])] for k in range(4)]

    def batch(views):
        r.rebinBatch(views)
        return [(r.readViewImage(v).view(np.uint16).copy(), *r.readViewRefs(v)) for v in range(2)]
    want = [batch(s) for s in sets]
    r.setCudaGraph(True)
    for k in (0, 1, 2, 3, 1, 0):
        for a, b in zip(batch(sets[k]), want[k]):
            for x, y in zip(a, b):
                assert np.array_equal(x, y), k


def test_blocks_handed_on_in_two_contexts(built_lib):
    p, lists = long_lists()
    rs = [make() for _ in range(2)]
    try:
        for r in rs:
            r.setSplatData(scenes.scene_small(N, seed=1))
            r.setTuning(16, 8, 0)
            r.setCamera(scenes.small_camera(W, H).getUniformData(W, H), W, H)
            r.writeBuffer("projected_splats", p)
            r.writeBuffer("tile_offsets",
                          np.cumsum([0] + [len(x) for x in lists]).astype(np.uint32))
            r.writeBuffer("sort_values_a", np.concatenate(lists).astype(np.uint32))
        rs[0].setSplitAllTiles(True)
        rs[0].rasterizeTiles()
        want = rs[0].readImage().view(np.uint16).copy()
        rs[0].setSplitAllTiles(False)
        errors, sent = [], [0, 0]

        def run(i):
            try:
                for _ in range(8):
                    for _ in range(4):
                        rs[i].rasterizeTiles()
                    rs[i].synchronize()
                    sent[i] += int(rs[i].readBuffer("raster_pool")[0])
                    if not np.array_equal(rs[i].readImage().view(np.uint16), want):
                        raise AssertionError(f"context {i}")
            except Exception as e:  # reported below, on the main thread
                errors.append(e)
        threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(300)
        assert not errors, errors
        assert min(sent) > 0
    finally:
        for r in rs:
            r.destroy()


@pytest.mark.parametrize("graphs", [(False,), (True,), (False, True), (True, False, False)])
def test_copies_under_way_while_the_next_frame_starts(renderer, graphs):
    torch = pytest.importorskip("torch")
    r = renderer
    w, h = 1920, 1080
    data = scenes.scene_small(60_000, seed=2)
    r.setSplatData(data)
    r.setTuning(16, 8, 0)
    us = [scenes.camera_at((0.5 * k - 1.0, 0.3, 6.0), w, h).getUniformData(w, h) for k in range(5)]
    want = []
    for u in us:
        r.rebin(data.splatCount, 120, 68, w, h, u)
        want.append(r.readImage().view(np.uint16).copy())
    out = torch.zeros(len(us) * 3, h, w, 4, dtype=torch.float16).pin_memory()
    for i in range(len(out)):
        r.setCudaGraph(graphs[i % len(graphs)])
        r.rebin(data.splatCount, 120, 68, w, h, us[i % 5], check=False)
        r._call("gs3d_copy_buffer_async", _lib.BUFFERS["splat_target"],
                C.c_void_p(out[i].data_ptr()), out[i].nbytes)
    r.synchronize()
    for i, img in enumerate(out):
        assert np.array_equal(img.numpy().view(np.uint16), want[i % 5]), i
