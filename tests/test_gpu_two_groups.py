"""Mixed filter on a mesh whose cells lie on both sides of the 128-row tile (125, 130 and 135 dofs): the group without
enrichment rows runs on the side stream.  Its tiles, built in the first fused step of an operator pair and again after
a reassembly, must be complete by then: the same bits as with the groups one after the other."""
import numpy as np
import pytest

import gbfe.enrichment as E
import gbfe.mesh as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem():
    return E.enriched_problem(4, 4, 12.0, 2, 6.0, 0.4, seed=3, keep_quadrature=True)


@pytest.mark.parametrize("m", [24, 64, 130])
def test_side_stream_group_reads_complete_tiles(gpu_ctx, problem, m):
    from gbfe import api

    p = problem
    assert p.nd_per_cell.min() == 125 and p.nd_per_cell.max() > 128
    q = p.extra["quad_cells"]
    X0, eig = M.random_block(p.n_dofs, m, 8), np.linspace(-2.0, 0.5, m)
    out = {}
    for split in (True, False):
        gpu_ctx.set_split_groups(split)
        try:
            basis = api.FEBasisManager.from_problem(gpu_ctx, p)
            Mo = api.CFEOverlapOperatorContext(basis, p.M, mixed=True)
            H = api.KohnShamOperatorContextFE(basis, p.H, mixed=True)
            inv = lambda: api.OrthoEFEOverlapInverseOpContextGLL(basis, p.m_gll_diag, p.extra["enr_begin"],  # noqa: E731
                                                                 p.extra["enr_block_inv"])
            X, Y = api.MultiVector(basis, m, init=X0), api.MultiVector(basis, m)
            Xf, Yf = api.MultiVector(basis, m, np.float32, X0.astype(np.float32)), api.MultiVector(basis, m, np.float32)
            H.apply(Xf, Yf)  # (creates the side stream)
            got = []
            for step in range(4):
                if step == 2:  # another potential on the same operator
                    api.assemble_cells(H, q["nq"], q["B"], 0.5 * q["w"], p.K, 0.5)
                Mi = inv()  # another operator pair: tiles of its own
                api.ResidualChebyshevFilterGEP(H, Mo, Mi, eig, X, 5, -6.0, 2.0, 300.0, Y, mixed=True)
                got.append(Y.numpy())
            gpu_ctx.check_status()
            out[split] = got
        finally:
            gpu_ctx.set_split_groups(True)
    assert all(np.isfinite(y).all() for y in out[True])
    assert np.abs(out[True][2] - out[True][1]).max() > 0.0
    for a, b in zip(out[True], out[False]):
        assert np.array_equal(a, b)
