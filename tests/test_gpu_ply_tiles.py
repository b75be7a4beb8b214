"""PLY decode at the edges of its staging: row counts around a block's rows,
bodies at every byte offset from a 16-byte boundary and ending where the buffer
ends, rows of few and of many properties, rows too wide to stage."""
import numpy as np
import pytest

from gs3d import GaussianSplatRenderer, Scene, ply, scenes
from oracle import ply_oracle

from test_gpu_ply import check_loaded

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer(built_lib):
    r = GaussianSplatRenderer(Scene())
    r.init()
    yield r
    r.destroy()


def load(r, raw, offset=0, **kw):
    data = ply.write_ply(raw, **kw)
    # an allocation of its own: the last row ends with it
    buf = np.frombuffer(b"\0" * offset + data, np.uint8)[offset:]
    r.loadPly(memoryview(buf))
    check_loaded(r, ply_oracle.load(data))


@pytest.mark.parametrize("n", [1, 127, 128, 129, 165, 166, 1000])
@pytest.mark.parametrize("deg", [0, 3])
@pytest.mark.parametrize("fmt", ["binary_little_endian", "binary_big_endian", "ascii"])
def test_row_counts(renderer, oracle, n, deg, fmt):
    load(renderer, scenes.raw_clusters(n, seed=n, sh_degree=deg), fmt=fmt)


@pytest.mark.parametrize("offset", range(16))
def test_byte_offsets(renderer, oracle, offset):
    load(renderer, scenes.raw_clusters(300, seed=5, sh_degree=1), offset,
         types={"f_dc_0": "uchar"})


@pytest.mark.parametrize("rest", [300, 9000, 12000])
def test_wide_rows(renderer, oracle, rest):
    raw = scenes.raw_clusters(5, seed=1, sh_degree=3)
    load(renderer, raw, f_rest_count=rest)
