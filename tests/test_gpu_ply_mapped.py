"""PLY loads from a memory-mapped file: whose pages nobody has read yet, again from
the same mapping, and with rows that start and end inside a page."""
import mmap

import pytest

from gs3d import GaussianSplatRenderer, Scene, ply, scenes
from oracle import ply_oracle

from test_gpu_ply import check_loaded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,deg,fmt", [(1, 0, "binary_little_endian"),
                                       (3000, 3, "binary_little_endian"),
                                       (20_000, 1, "binary_big_endian")])
def test_load_from_a_mapped_file(built_lib, oracle, tmp_path, n, deg, fmt):
    data = ply.write_ply(scenes.raw_clusters(n, seed=n, sh_degree=deg), fmt)
    path = tmp_path / "scene.ply"
    path.write_bytes(data)
    want = ply_oracle.load(data)
    r = GaussianSplatRenderer(Scene())
    r.init()
    try:
        for _ in range(3):  # a new mapping each time
            with open(path, "rb") as f:
                rows = memoryview(mmap.mmap(f.fileno(), 0, access=mmap.ACCESS_READ))
            for _ in range(2):
                r.loadPly(rows)
                check_loaded(r, want)
    finally:
        r.destroy()
