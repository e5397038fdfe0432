"""The m x m block of a fused pass above the host's range (own Cholesky factor and triangular solves): after one pass the
block is M-orthonormal and diagonalises H.  Sizes at the edges of the 32-column panels and of the range.

Bound: 4 m 2^-52 cond, with cond <= 1e4 for the overlap of a degree-2 filtered random block (growth below 2 on the
wanted interval, overlap weights within 64, random block of at least 4 m rows or m rows of a well separated subspace)."""
import numpy as np
import pytest

import gbfe.mesh as M
from gbfe._lib import STATUS_NAMES
from test_gpu_parity import _setup

pytestmark = pytest.mark.gpu


def one_pass(ctx, p, X0):
    from gbfe import api

    basis, H, Mo, Mi, s, oH, oM, oMi = _setup(ctx, p)
    b = s.lanczos_bounds(oH, oM, oMi)
    lo, hi = b[0], b[1] + b[2] / 10
    m = X0.shape[1]
    X = api.MultiVector(basis, m, init=X0)
    solver = api.KohnShamEigenSolver(m // 2, 2, 1, 1e-9, bounds=(lo, lo + 0.1 * (hi - lo), hi), fixed_passes=True)
    rc, eig, _, _ = solver.solve(H, X, Mo, Mi)
    HX, MX = api.MultiVector(basis, m), api.MultiVector(basis, m)
    H.apply(X, HX)
    Mo.apply(X, MX)
    return rc, eig, X.numpy(), HX.numpy(), MX.numpy(), max(abs(lo), abs(hi))


@pytest.fixture(scope="module")
def boxes():
    return {n: M.ks_box(n, 3, 8.0, 2, 4.0, 0.5, seed=11) for n in (5, 6)}


@pytest.mark.parametrize("m", [128, 129, 159, 160, 161, 255, 256, 257, 1024, 1025])
def test_pass_orthonormal_and_diagonal(gpu_ctx, boxes, m):
    p = boxes[6 if m > 300 else 5]
    rc, eig, X, HX, MX, top = one_pass(gpu_ctx, p, M.random_block(p.n_dofs, m, m))
    assert np.all(np.diff(eig) >= 0)
    tol = 4 * m * 2.0 ** -52 * 1e4
    assert np.abs(X.T @ MX - np.eye(m)).max() <= tol
    assert np.abs(X.T @ HX - np.diag(eig)).max() <= tol * top


def test_singular_overlap_is_an_error(gpu_ctx, boxes):
    X0 = M.random_block(boxes[5].n_dofs, 200, 3)
    X0[:, 150] = 0.0
    rc = one_pass(gpu_ctx, boxes[5], X0)[0]
    assert STATUS_NAMES[rc] in ("ERR_LAPACK", "ERR_NOT_ORTHONORMALIZABLE")
