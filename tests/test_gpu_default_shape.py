"""Default launch shape of the split-BF16 cell product (no tuned entry): block widths on both sides of every line of
the rule, for cells of one (125 dofs) and two (216 dofs) row tiles, within TC_TOL (1e-4 relative max-norm, the
split-BF16 product's bound) of the FP64 apply."""
import numpy as np
import pytest

import gbfe.mesh as M
from conftest import rel_maxnorm

TC_TOL = 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("degree", [2, 4, 5])
@pytest.mark.parametrize("m", [1, 16, 31, 32, 33, 36, 48, 49, 52, 129])
def test_default_shape_matches_fp64(gpu_ctx, degree, m):
    from gbfe import api

    prob = M.ks_box(2, degree, 8.0, 1, 4.0, 0.5, seed=46)
    X0 = M.random_block(prob.n_dofs, m, 10)
    basis = api.FEBasisManager.from_problem(gpu_ctx, prob)
    H = api.KohnShamOperatorContextFE(basis, prob.H, mixed=True)
    Y, Yf = api.MultiVector(basis, m), api.MultiVector(basis, m, dtype=np.float32)
    H.apply(api.MultiVector(basis, m, init=X0), Y)
    H.apply(api.MultiVector(basis, m, dtype=np.float32, init=X0.astype(np.float32)), Yf)
    gpu_ctx.check_status()
    assert rel_maxnorm(Yf.numpy(), Y.numpy()) <= TC_TOL
