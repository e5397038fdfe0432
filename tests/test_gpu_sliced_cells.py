"""FP64-accurate sliced cell product: cells at the edges of its 128-row tiles and 32-row K chunks, widths at the edges of
its 64-vector tiles and of the pairs of tiles that share matrix slices, rows and columns of very different size.

Bound: the FP64 apply's 1e-12 relative max-norm against the FP64 FMA product; for the scaled inputs, per entry, K 2^-52
max|a_row| max|x_col| (a 55-bit fixed point per matrix row and vector: two roundings of 2^-56 and dropped products
below 2^-54 of that per term, added over K terms)."""
import numpy as np
import pytest

import gbfe.mesh as M
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


def both(ctx, basis, mats, X0):
    from gbfe import api

    m, out = X0.shape[1], []
    for mode in (0, 1):
        H = api.KohnShamOperatorContextFE(basis, mats, fp64_tensor=bool(mode))
        ctx.set_fp64_apply(mode)
        try:
            Y = api.MultiVector(basis, m)
            H.apply(api.MultiVector(basis, m, init=X0), Y)
            out.append(Y.numpy())
        finally:
            ctx.set_fp64_apply(0)
    ctx.check_status()
    return out


@pytest.mark.parametrize("nd", [1, 8, 31, 32, 33, 65, 127, 128, 129, 216, 255, 256])
@pytest.mark.parametrize("m", [1, 64, 65, 130])
def test_sizes(gpu_ctx, nd, m):
    from gbfe import api

    rng = np.random.default_rng(nd * 1000 + m)
    cells, N = 9, 5 * nd + 3
    ids = np.concatenate([rng.permutation(N)[:nd] for _ in range(cells)]).astype(np.uint32)
    basis = api.FEBasisManager(gpu_ctx, np.full(cells, nd, np.uint32), ids, N)
    ref, got = both(gpu_ctx, basis, rng.standard_normal(cells * nd * nd), rng.standard_normal((N, m)))
    assert rel_maxnorm(got, ref) <= 1e-12


@pytest.mark.parametrize("m", [3, 256, 321])
def test_mixed_sizes_and_scales(gpu_ctx, m):
    """Cells of one and of two row tiles in one mesh (disjoint dofs); rows and vectors scaled over 40 decades."""
    from gbfe import api

    rng = np.random.default_rng(m)
    nd = np.array([27, 216, 64, 125, 200, 27, 216], np.uint32)
    off = np.concatenate([[0], np.cumsum(nd.astype(np.int64))])
    N = int(off[-1])
    basis = api.FEBasisManager(gpu_ctx, nd, np.arange(N, dtype=np.uint32), N)
    A = [rng.standard_normal((n, n)) * 10.0 ** rng.uniform(-20, 20, (n, 1)) for n in nd]  # y_j = sum_k A[j, k] x_k
    X0 = rng.standard_normal((N, m)) * 10.0 ** rng.uniform(-20, 20, (1, m))
    ref, got = both(gpu_ctx, basis, np.concatenate([a.ravel() for a in A]), X0)
    xmax = np.abs(X0).max(0)
    for c, n in enumerate(nd):
        rows = slice(off[c], off[c + 1])
        bound = int(n) * 2.0 ** -52 * np.abs(A[c]).max(1)[:, None] * xmax[None]
        assert np.all(np.abs(got[rows] - ref[rows]) <= bound)
