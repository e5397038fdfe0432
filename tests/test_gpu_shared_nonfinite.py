"""Batched CG from starts that are not finite, or overflow: the tensor-core product of shared matrices ends every
instance as the FMA product of the same cells does (status, iteration and kind of the residual)."""
import numpy as np
import pytest

import gbfe.poisson as P

pytestmark = pytest.mark.gpu


def outcome(api, basis, K, pb, x0, b):
    x = api.MultiVector(basis, 1, init=x0[:, None])
    its, status, rn = api.pcg_solve_batched(K, api.PreconditionerJacobi(basis, pb.jacobi_diag),
                                            api.MultiVector(basis, 1, init=b[:, None]), x, pb.inst_dof_off, 40, 1e-300,
                                            1e-10, 1e10)
    kind = np.where(np.isnan(rn), 2, np.isinf(rn))
    return list(its), list(status), list(kind), np.isnan(x.numpy()).any(), np.isinf(x.numpy()).any()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e308, 1e-310])
@pytest.mark.parametrize("where", ["x", "b"])
def test_same_outcome_as_the_fma_product(gpu_ctx, value, where):
    from gbfe import api

    pb = P.batch(count=2, seed=5, n_range=(9, 9), degrees=(3,))
    assert int((pb.nd_per_cell[: 9 ** 3].astype(np.int64) ** 2).sum()) >= 2_000_000
    basis = api.FEBasisManager(gpu_ctx, pb.nd_per_cell, pb.cell_dof_ids, pb.n_dofs, pb.constraints)
    nd = int(pb.nd_per_cell[0])
    tensor = api.IndexedCellMatrixOperatorContext(basis, pb.mats, pb.cell_to_mat)
    fma = api.LaplaceOperatorContextFE(basis, np.tile(pb.mats[: nd * nd], pb.nd_per_cell.size))
    free = np.setdiff1d(np.arange(int(pb.inst_dof_off[1])), pb.constraints.row_ids)
    x0, b = np.zeros(pb.n_dofs), pb.b.copy()
    (x0 if where == "x" else b)[free[len(free) // 2]] = value  # in the first instance
    got, ref = outcome(api, basis, tensor, pb, x0, b), outcome(api, basis, fma, pb, x0, b)
    assert got == ref
    gpu_ctx.check_status()
