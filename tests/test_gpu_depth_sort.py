"""The fused rebin's depth order against the six reference stages, bit for bit:
splat counts around its 5120-key partitions, depths whose keys span less than
2^27 (three 9-bit passes) and more (four 8-bit passes), equal depths, everything
culled but one."""
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


def frame(r, data, u, w, h, stagewise):
    r.setStagewise(stagewise)
    r.rebin(data.splatCount, -(-w // 16), -(-h // 16), w, h, u)
    r.setStagewise(False)
    R = r.refCount()
    return (R, r.readBuffer("sort_keys_a", R), r.readBuffer("sort_values_a", R),
            r.readBuffer("tile_offsets"))


def along_the_view(n, near, far, seed):
    """Splats in a cone before a camera at the origin looking down -z."""
    rng = np.random.default_rng(seed)
    z = np.exp(rng.uniform(np.log(near), np.log(far), n))
    xy = rng.uniform(-0.4, 0.4, (n, 2)) * z[:, None]
    size = np.log(z[:, None] * rng.uniform(1e-3, 1e-2, (n, 3)))
    return scenes.activate(np.concatenate([xy, -z[:, None]], 1), rng.normal(0, 0.5, (n, 3)),
                           rng.normal(0, 1.5, n), size, rng.standard_normal((n, 4)))


@pytest.mark.parametrize("n", [1, 31, 5119, 5120, 5121, 10_240, 92_161])
@pytest.mark.parametrize("near,far", [(1.0, 1.0), (2.0, 60.0), (1e-3, 60.0), (1e-3, 5e3)])
def test_order_equals_the_reference_stages(renderer, n, near, far):
    r = renderer
    w, h = 400, 300
    data = along_the_view(n, near, far, n)
    u = scenes.camera_at((0.0, 0.0, 0.0), w, h, target=(0.0, 0.0, -1.0), near=1e-4,
                         far=1e5).getUniformData(w, h)
    r.setSplatData(data)
    want = frame(r, data, u, w, h, True)
    lo = want[1][:, 1]
    assert want[0] > 0
    if n > 1000 and far / near > 2 ** 17:
        assert int(lo.max()) - int(lo.min()) >= 2 ** 27
    got = frame(r, data, u, w, h, False)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [2047, 2048, 2049, 130_000, 311_296, 311_297])
def test_order_at_the_partition_sizes(renderer, n):
    """Partitions of 2048 keys up to 311,296 splats, then of 5120."""
    r = renderer
    w, h = 640, 480
    data = along_the_view(n, 2.0, 60.0, n)
    u = scenes.camera_at((0.0, 0.0, 0.0), w, h, target=(0.0, 0.0, -1.0)).getUniformData(w, h)
    r.setSplatData(data)
    want = frame(r, data, u, w, h, True)
    got = frame(r, data, u, w, h, False)
    assert want[0] > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_one_splat_among_culled_ones(renderer):
    r = renderer
    w, h = 400, 300
    data = along_the_view(20_000, 2.0, 60.0, 7)
    data.positions[:, 2] *= -1.0
    data.positions[12_345, 2] *= -1.0
    u = scenes.camera_at((0.0, 0.0, 0.0), w, h, target=(0.0, 0.0, -1.0)).getUniformData(w, h)
    r.setSplatData(data)
    want = frame(r, data, u, w, h, True)
    got = frame(r, data, u, w, h, False)
    assert want[0] > 0 and set(want[2]) == {12_345}
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
