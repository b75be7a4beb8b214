"""The cost model's training kernels at the edges of their 64-sample tiles:
forward and backward against the float64 oracle, on unaligned buffers."""
import ctypes as C

import numpy as np
import pytest

from gs3d import _lib, learned
from oracle import mlp_oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def shifted(a, by):
    """A device copy that starts `by` floats into its allocation."""
    t = torch.empty(a.size + by, device="cuda")[by:]
    t.copy_(torch.from_numpy(np.ascontiguousarray(a).reshape(-1)))
    return t


@pytest.mark.parametrize("n", [1, 63, 64, 65, 300, 64 * 304, 64 * 304 + 1, 50_011])
def test_forward_and_backward_match_the_oracle(built_lib, n):
    lib = _lib.load()
    rng = np.random.default_rng(n)
    p = learned.init_params(3, 0.7)
    p[1024:1088] = rng.normal(0, 0.1, 64)
    x = rng.normal(0, 1, (n, 16)).astype(np.float32)
    t = rng.normal(2, 1, n).astype(np.float32)
    dp, dx, dt = shifted(p, 1), shifted(x, 3), shifted(t, 1)
    acts = torch.full((n * 129 + 1,), 7.0, device="cuda")[1:]
    y = torch.empty(n, device="cuda")
    g = torch.zeros(len(p) + 1, device="cuda")[1:]
    dev = lambda a: C.c_void_p(a.data_ptr())  # noqa: E731
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.gs3d_mlp_forward(dev(dp), dev(dx), n, dev(acts), dev(y), s) == 0
    assert lib.gs3d_mlp_backward(dev(dp), dev(dx), dev(acts), dev(dt), n, dev(g), s) == 0
    torch.cuda.synchronize()
    y_ref, h1, h2 = mlp_oracle.forward(p, x)
    a = acts.cpu().numpy().reshape(n, 129)
    # sums of at most 64 products and a bias, three layers deep: 200 roundings
    tol = 200 * 2.0 ** -24
    want = np.concatenate([h1, h2, y_ref[:, None]], 1)
    big = np.abs(want).max()
    assert np.abs(a - want).max() <= tol * 64 * big
    assert np.array_equal(a[:, 128], y.cpu().numpy())
    g_ref = mlp_oracle.grad(p, x, t)
    # n terms in any order, each itself a chain as above
    assert np.abs(g.cpu().numpy() - g_ref).max() <= 1e-3 * np.abs(g_ref).max() + 1e-6
