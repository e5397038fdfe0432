"""FP64 FMA apply: narrow blocks (four lanes per column), Dirichlet rows masked in the gather and zeroed in X by the
assembly, vectors on 8-byte boundaries, and the two-launch FP64 filter step."""
import ctypes as C

import numpy as np
import pytest

import gbfe.mesh as M
from oracle import oracle as O
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 2, 3, 5])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5])
def test_narrow_apply_and_masked_rows(gpu_ctx, degree, m):
    """1e-12 relative max-norm of the oracle's apply (the FP64 bar); a NaN on a Dirichlet row of X reads as zero."""
    from gbfe import api

    p = M.ks_box(3, degree, 8.0, 2, 4.0, 0.5, seed=12)
    basis = api.FEBasisManager.from_problem(gpu_ctx, p)
    H = api.KohnShamOperatorContextFE(basis, p.H)
    s = O.OracleSystem.from_problem(p)
    X0 = M.random_block(p.n_dofs, m, 3 + m)
    Xn = X0.copy()
    Xn[p.constraints.row_ids[::2]] = np.nan
    X, Y = api.MultiVector(basis, m, init=Xn), api.MultiVector(basis, m)
    H.apply(X, Y)
    Xo = X0.copy()
    Yo = s.apply(s.cell_op(p.H), Xo)
    assert rel_maxnorm(Y.numpy(), Yo) <= 1e-12
    assert np.array_equal(X.numpy(), Xo)


@pytest.mark.parametrize("m", [4, 6])
def test_wrapped_vectors_off_16_byte_boundaries(gpu_ctx, small_problem, m):
    """X, Y at 8-byte boundaries give the bits of aligned ones."""
    import torch
    from gbfe import api

    p = small_problem
    basis = api.FEBasisManager.from_problem(gpu_ctx, p)
    H = api.KohnShamOperatorContextFE(basis, p.H)
    X0 = M.random_block(p.n_dofs, m, 5)
    Xa, Ya = api.MultiVector(basis, m, init=X0), api.MultiVector(basis, m)
    H.apply(Xa, Ya)
    raw = [torch.zeros(p.n_dofs * m + 1, dtype=torch.float64, device="cuda") for _ in range(2)]
    raw[0][1:] = torch.from_numpy(X0.ravel()).cuda()
    torch.cuda.synchronize()
    h = []
    for t in raw:
        v = C.c_void_p()
        assert gpu_ctx.lib.gbfe_mv_wrap(basis.h, m, 0, C.c_void_p(t[1:].data_ptr()), C.byref(v)) == 0
        h.append(v)
    assert gpu_ctx.lib.gbfe_apply(H.h, h[0], h[1]) == 0
    gpu_ctx.synchronize()
    assert np.array_equal(raw[1][1:].cpu().numpy().reshape(-1, m), Ya.numpy())
    assert np.array_equal(raw[0][1:].cpu().numpy().reshape(-1, m), Xa.numpy())
    for v in h:
        gpu_ctx.lib.gbfe_mv_destroy(v)


@pytest.mark.parametrize("m", [1, 5, 8])
def test_fused_fp64_filter_step(gpu_ctx, small_problem, m):
    """The same products and sums as the separate launches: 1e-13 relative (only the contraction of the step's
    multiply-adds may differ)."""
    from gbfe import api

    p = small_problem
    basis = api.FEBasisManager.from_problem(gpu_ctx, p)
    H = api.KohnShamOperatorContextFE(basis, p.H)
    Mo = api.CFEOverlapOperatorContext(basis, p.M)
    Mi = api.CFEOverlapInverseOpContextGLL(basis, p.m_gll_diag)
    X0, eig = M.random_block(p.n_dofs, m, 6), np.linspace(-3.0, 0.5, m)
    out = []
    for fused in (True, False):
        gpu_ctx.set_fused_filter(fused)
        try:
            X, Y = api.MultiVector(basis, m, init=X0), api.MultiVector(basis, m)
            api.ResidualChebyshevFilterGEP(H, Mo, Mi, eig, X, 7, -4.0, 2.0, 60.0, Y)
            out.append(Y.numpy())
        finally:
            gpu_ctx.set_fused_filter(True)
    assert rel_maxnorm(out[0], out[1]) <= 1e-13
