"""Accuracy of the m x m stages of a fused pass above the host's range (Cholesky factor, triangular solves, refined
eigenproblem), against LAPACK on the same projected matrices: the filtered block Y comes from the public filter, its
overlap's condition number is computed, and the pass's orthogonality and diagonality may be 8 times those of the block
that scipy's factor and solves give (each an accumulation of m rounded products, in another order), or of m 2^-53
where that is smaller.  Eigenvalues: 4 m 2^-52 cond of the largest."""
import numpy as np
import pytest
import scipy.linalg as sla

import gbfe.mesh as M
from test_gpu_parity import _setup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def box():
    return M.ks_box(6, 3, 8.0, 2, 4.0, 0.5, seed=11)


@pytest.mark.parametrize("m", [129, 160, 255, 256, 512, 1024])
def test_pass_is_as_accurate_as_lapack(gpu_ctx, box, m):
    from gbfe import api

    basis, H, Mo, Mi, s, oH, oM, oMi = _setup(gpu_ctx, box)
    b = s.lanczos_bounds(oH, oM, oMi)
    lo, hi = b[0], b[1] + b[2] / 10
    bounds = (lo, lo + 0.1 * (hi - lo), hi)
    X0 = M.random_block(box.n_dofs, m, m)

    def products(Z):
        X, HX, MX = api.MultiVector(basis, m, init=Z), api.MultiVector(basis, m), api.MultiVector(basis, m)
        H.apply(X, HX)
        Mo.apply(X, MX)
        Z = X.numpy()
        return Z.T @ MX.numpy(), Z.T @ HX.numpy()

    X, Y = api.MultiVector(basis, m, init=X0), api.MultiVector(basis, m)
    api.ResidualChebyshevFilterGEP(H, Mo, Mi, np.zeros(m), X, 2, *bounds, Y)
    Yh = Y.numpy()
    SM, SH = products(Yh)
    SM, SH = 0.5 * (SM + SM.T), 0.5 * (SH + SH.T)
    cond = np.linalg.cond(SM)
    L = np.linalg.cholesky(SM)
    Hp = sla.solve_triangular(L, sla.solve_triangular(L, SH, lower=True).T, lower=True)
    w, V = np.linalg.eigh(0.5 * (Hp + Hp.T))
    ref_m, ref_h = products(Yh @ sla.solve_triangular(L, V, lower=True, trans="T"))

    X = api.MultiVector(basis, m, init=X0)
    rc, eig, _, _ = api.KohnShamEigenSolver(m // 2, 2, 1, 1e-9, bounds=bounds, fixed_passes=True).solve(H, X, Mo, Mi)
    got_m, got_h = products(X.numpy())
    top = np.abs(w).max()
    eye, unit = np.eye(m), m * 2.0 ** -53
    assert np.abs(got_m - eye).max() <= 8 * max(np.abs(ref_m - eye).max(), unit)
    assert np.abs(got_h - np.diag(eig)).max() <= 8 * max(np.abs(ref_h - np.diag(w)).max(), unit * top)
    assert np.abs(np.asarray(eig) - w).max() <= 4 * m * 2.0 ** -52 * cond * top
