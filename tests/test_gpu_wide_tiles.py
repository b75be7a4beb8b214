"""Tiles of more than 1024 pixels are for the fused rebin: gs3d_rebin_batch, which
is always fused, takes them whatever the flags; the stage entry points refuse them."""
import numpy as np
import pytest

from gs3d import GaussianSplatRenderer, Gs3dError, Scene, _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_stage_entry_points_and_batches_at_wide_tiles(built_lib, graph):
    data = scenes.scene_small(30_000, seed=6)
    w, h = 640, 360
    u = scenes.small_camera(w, h).getUniformData(w, h)
    r = GaussianSplatRenderer(Scene())
    r.init()
    try:
        r.setSplatData(data)
        r.setTuning((64, 32), 8, 0)
        r.setCudaGraph(graph)
        r.rebinBatch([(0, u, w, h)])
        want = r.readViewImage(0).view(np.uint16).copy()
        r.setStagewise(True)
        r.rebinBatch([(0, u, w, h)])
        assert np.array_equal(r.readViewImage(0).view(np.uint16), want)
        for stagewise in (True, False):
            r.setStagewise(stagewise)
            with pytest.raises(Gs3dError) as ei:
                r.rasterizeTiles()
            assert ei.value.code == _lib.ERR_INVALID_ARG
    finally:
        r.destroy()
