"""Column dots and norms: the one-launch kernel for narrow blocks and the two-stage one, at the edges of their column
groups and of the batches of eight rows, against extended precision.

Bound per column: N 2^-53 sum|x y| (N rounded additions), relative for the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 31, 32, 33, 64, 100, 255, 256, 257, 512])
@pytest.mark.parametrize("cells", [1, 37, 700])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_dots(gpu_ctx, m, cells, dtype):
    from gbfe import api

    nd = 8
    N = cells * nd
    rng = np.random.default_rng(m + cells)
    basis = api.FEBasisManager(gpu_ctx, np.full(cells, nd, np.uint32), np.arange(N, dtype=np.uint32), N)
    x, y = (rng.standard_normal((N, m)).astype(dtype) for _ in range(2))
    X, Y = api.MultiVector(basis, m, dtype=dtype, init=x), api.MultiVector(basis, m, dtype=dtype, init=y)
    xl, yl = x.astype(np.longdouble), y.astype(np.longdouble)
    ref = (xl * yl).sum(0)
    tol = N * 2.0 ** -53
    assert np.all(np.abs(X.dot(Y) - ref) <= tol * np.abs(xl * yl).sum(0))
    norms = np.sqrt((xl * xl).sum(0))
    assert np.all(np.abs(X.l2Norms() - norms) <= tol * norms)
