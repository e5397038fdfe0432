"""Blocks of more vectors than a full grid has threads (622,592 on 152 SMs): the fused steps of the FP64 filter and the
assembly of an apply still reach every column.  One cell of 8 dofs; the filter against the separate launches (the same
operations), the apply against the dense product (8 products and sums per entry: 16 2^-53 of sum |a||x|)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [622_593, 700_000])
def test_every_column_is_reached(gpu_ctx, m):
    from gbfe import api

    rng = np.random.default_rng(m)
    A = rng.standard_normal((8, 8))
    A = A + A.T
    basis = api.FEBasisManager(gpu_ctx, np.array([8], np.uint32), np.arange(8, dtype=np.uint32), 8)
    H = api.KohnShamOperatorContextFE(basis, A.ravel())
    Mo = api.CFEOverlapOperatorContext(basis, np.eye(8).ravel())
    Mi = api.CFEOverlapInverseOpContextGLL(basis, np.ones(8))
    X0 = rng.standard_normal((8, m))
    X, Y = api.MultiVector(basis, m, init=X0), api.MultiVector(basis, m)
    H.apply(X, Y)
    assert np.all(np.abs(Y.numpy() - A @ X0) <= 16 * 2.0 ** -53 * (np.abs(A) @ np.abs(X0)))
    eig, out = np.linspace(-2.0, 2.0, m), []
    for fused in (True, False):
        gpu_ctx.set_fused_filter(fused)
        try:
            api.ResidualChebyshevFilterGEP(H, Mo, Mi, eig, X, 4, -10.0, 1.0, 12.0, Y)
            out.append(Y.numpy())
        finally:
            gpu_ctx.set_fused_filter(True)
    gpu_ctx.check_status()
    scale = np.abs(out[1]).max()
    assert np.isfinite(scale) and np.abs(out[0] - out[1]).max() <= 1e-13 * scale
