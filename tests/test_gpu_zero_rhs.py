"""Batched CG with right-hand sides of zero: such an instance is done at iteration 0 with x = 0 and a zero residual, and
leaves the others alone -- with the tensor-core product of shared matrices and with the FMA product."""
import numpy as np
import pytest

import gbfe.poisson as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 9])  # 0.26 and 3.0 M matrix entries an instance
def test_zero_right_hand_side(gpu_ctx, n):
    from gbfe import api

    pb = P.batch(count=3, seed=2, n_range=(n, n), degrees=(3,))
    basis = api.FEBasisManager(gpu_ctx, pb.nd_per_cell, pb.cell_dof_ids, pb.n_dofs, pb.constraints)
    K = api.IndexedCellMatrixOperatorContext(basis, pb.mats, pb.cell_to_mat)
    J = api.PreconditionerJacobi(basis, pb.jacobi_diag)
    off = pb.inst_dof_off
    b0 = pb.b.copy()
    b0[int(off[1]):int(off[2])] = 0.0
    out = {}
    for name, rhs in (("zero", b0), ("full", pb.b)):
        x = api.MultiVector(basis, 1)
        its, status, rn = api.pcg_solve_batched(K, J, api.MultiVector(basis, 1, init=rhs[:, None]), x, off, 1000, 1e-14,
                                                1e-10, 1e10)
        out[name] = np.asarray(its), np.asarray(status), np.asarray(rn), x.numpy()[:, 0]
    its, status, rn, x = out["zero"]
    assert status[1] == 0 and its[1] == 0 and rn[1] == 0.0
    assert not x[int(off[1]):int(off[2])].any()
    for i in (0, 2):
        d = slice(int(off[i]), int(off[i + 1]))
        assert status[i] == 0 and its[i] == out["full"][0][i] and np.array_equal(x[d], out["full"][3][d])
