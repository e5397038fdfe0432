"""One-vector tensor-core product of operators whose cells share matrices, inside
the batched CG solve: cell sizes and counts at the edges of its 32-row K chunks,
128-row tiles and 64-cell items, several matrices at once, and non-finite input.

Every cell is a system of its own here (disjoint dofs, one SPD matrix per size
with eigenvalues in [1, 10]), so the exact solution is a dense solve.  Bound: the
solver stops at |r| <= tol |b| per instance, so |x - x*| <= |A^-1| tol |b| = tol
|b|; twice that covers the recurrence's drift from the true residual.
"""
import numpy as np
import pytest

TOL = 1e-12


def spd(n, rng):
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * rng.uniform(1.0, 10.0, n)) @ q.T
    return 0.5 * (a + a.T)


def disjoint(ctx, sizes, counts, rng):
    from gbfe import api

    c2m = np.repeat(np.arange(len(sizes), dtype=np.uint32), counts)
    rng.shuffle(c2m)
    nd = np.array(sizes, np.uint32)[c2m]
    off = np.concatenate([[0], np.cumsum(nd.astype(np.int64))])
    N = int(off[-1])
    mats = [spd(n, rng) for n in sizes]
    basis = api.FEBasisManager(ctx, nd, rng.permutation(N).astype(np.uint32), N)
    K = api.IndexedCellMatrixOperatorContext(basis, np.concatenate([a.ravel() for a in mats]), c2m)
    J = api.PreconditionerJacobi(basis, np.ones(N))
    return basis, K, J, mats, c2m, off


@pytest.mark.gpu
@pytest.mark.parametrize("sizes, counts", [
    ((128,), (385,)),                            # the largest cell, a last item of one cell
    ((127, 125, 96), (190, 191, 64)),            # below the tile, 32-row chunk multiples
    ((97, 64, 33, 32, 31), (700, 65, 63, 1, 130)),  # one row past a chunk, whole and nearly empty items
    ((100, 8, 7, 1), (640, 64, 3, 1)),           # very small cells beside large ones
])
def test_cells_solve_their_own_systems(gpu_ctx, sizes, counts):
    from gbfe import api

    assert sum(n * n * c for n, c in zip(sizes, counts)) >= 6_000_000  # the product under test runs
    rng = np.random.default_rng(sum(sizes))
    basis, K, J, mats, c2m, off = disjoint(gpu_ctx, sizes, counts, rng)
    b0 = rng.standard_normal(off[-1])
    b, x = api.MultiVector(basis, 1, init=b0[:, None]), api.MultiVector(basis, 1)
    its, status, rn = api.pcg_solve_batched(K, J, b, x, np.array([0, off[-1]], np.uint64), 400, 1e-300, TOL, 1e30)
    assert status[0] == 0 and its[0] > 5
    ids, xs, nb = basis._ids, x.numpy()[:, 0], np.linalg.norm(b0)
    for u, a in enumerate(mats):
        at = np.stack([ids[off[c]:off[c + 1]] for c in np.flatnonzero(c2m == u)])
        exact = np.linalg.solve(a, b0[at].T).T
        assert np.abs(xs[at] - exact).max() <= 2 * TOL * nb
    gpu_ctx.check_status()


@pytest.mark.gpu
def test_instances_stop_on_their_own_and_nan_stays_in_its_instance(gpu_ctx):
    """Three instances of 64-dof cells (mesh order): one converges at once (b = 0), one holds a NaN, one is sound."""
    from gbfe import api

    rng = np.random.default_rng(4)
    n, per = 64, 500
    a = spd(n, rng)
    N = 3 * per * n
    basis = api.FEBasisManager(gpu_ctx, np.full(3 * per, n, np.uint32), np.arange(N, dtype=np.uint32), N)
    K = api.IndexedCellMatrixOperatorContext(basis, a.ravel(), np.zeros(3 * per, np.uint32))
    b0 = rng.standard_normal(N)
    b0[:per * n] = 0.0
    b0[per * n + 77] = np.nan
    b, x = api.MultiVector(basis, 1, init=b0[:, None]), api.MultiVector(basis, 1)
    off = np.array([0, per * n, 2 * per * n, N], np.uint64)
    its, status, rn = api.pcg_solve_batched(K, api.PreconditionerJacobi(basis, np.ones(N)), b, x, off, 200, 1e-300, TOL,
                                            1e30)
    xs = x.numpy()[:, 0].reshape(3, per, n)
    assert status[2] == 0 and status[1] != 0
    assert np.all(xs[0] == 0.0) or np.isnan(xs[0]).all()  # 0 / 0 in the first step, as a CG on b = 0 does
    assert np.isnan(xs[1]).any()
    exact = np.linalg.solve(a, b0[2 * per * n:].reshape(per, n).T).T
    assert np.abs(xs[2] - exact).max() <= 2 * TOL * np.linalg.norm(b0[2 * per * n:])


@pytest.mark.gpu
def test_start_vector_with_values_on_dirichlet_rows(gpu_ctx):
    """The residual of iteration 0 goes through the product too: a random start, not zero on the Dirichlet rows, ends
    with them at zero and with the true residual (general apply) within twice the requested one per instance."""
    import gbfe.poisson as P
    from gbfe import api

    tol = 1e-9
    pb = P.batch(count=6, seed=8, n_range=(5, 6), degrees=(4,))
    assert sum(int(n) ** 2 for n in pb.nd_per_cell) >= 6_000_000
    basis = api.FEBasisManager(gpu_ctx, pb.nd_per_cell, pb.cell_dof_ids, pb.n_dofs, pb.constraints)
    K = api.IndexedCellMatrixOperatorContext(basis, pb.mats, pb.cell_to_mat)
    b = api.MultiVector(basis, 1, init=pb.b[:, None])
    x = api.MultiVector(basis, 1, init=np.random.default_rng(3).standard_normal((pb.n_dofs, 1)))
    its, status, rn = api.pcg_solve_batched(K, api.PreconditionerJacobi(basis, pb.jacobi_diag), b, x, pb.inst_dof_off,
                                            3000, 1e-300, tol, 1e10)
    xs, w = x.numpy()[:, 0], api.MultiVector(basis, 1)
    assert np.all(np.asarray(status) == 0) and np.all(xs[pb.constraints.row_ids] == 0.0)
    K.apply(x, w)
    r = pb.b - w.numpy()[:, 0]
    for i in range(pb.n_inst):
        d = slice(int(pb.inst_dof_off[i]), int(pb.inst_dof_off[i + 1]))
        assert np.linalg.norm(r[d]) <= 2 * tol * np.linalg.norm(pb.b[d])
