"""Batched CG: an instance's solution, iteration count and residual are bitwise those of its solve alone, whatever else
is in the batch -- instances below and above the size at which the cell products go to the tensor cores, and neighbours
that would change the path of the whole batch (a hanging row, matrices of their own per cell, cells of 150 dofs)."""
import numpy as np
import pytest

import gbfe.mesh as M
import gbfe.poisson as P

pytestmark = pytest.mark.gpu
LINE = 2_000_000  # expanded matrix entries from which an instance's products run on the tensor cores


def spd(n, rng):
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    return (q * rng.uniform(1.0, 10.0, n)) @ q.T


def instances():
    pb = P.batch(count=5, seed=24, n_range=(5, 11), degrees=(3, 4))
    out = []
    for i in range(pb.n_inst):
        v = P.instance_view(pb, i)
        nd0 = int(v["nd"][0])
        out.append(dict(nd=v["nd"], ids=v["ids"], N=v["N"], rows=v["cons"].row_ids, hang=None, b=v["b"], diag=v["diag"],
                        mats=[v["K"][:nd0 * nd0]], c2m=np.zeros(v["nd"].size, np.int64)))
    return out


def neighbour(kind, insts, rng):
    """One more instance for the batch."""
    if kind == "hanging row":
        n = dict(insts[0])
        free = np.setdiff1d(np.arange(n["N"]), n["rows"])
        r, a, b = (int(x) for x in rng.choice(free, 3, replace=False))
        return {**n, "hang": (r, (a, b), (0.5, 0.5)), "b": np.where(np.arange(n["N"]) == r, 0.0, n["b"])}
    nd = 64 if kind == "own matrices" else 150
    cells = 700 if kind == "own matrices" else 40
    mats = [spd(nd, rng).ravel() for _ in range(cells if kind == "own matrices" else 1)]
    N = nd * cells
    return dict(nd=np.full(cells, nd, np.uint32), ids=np.arange(N, dtype=np.uint32), N=N, rows=np.zeros(0, np.int64),
                hang=None, b=rng.standard_normal(N), diag=np.ones(N), mats=mats,
                c2m=np.arange(cells) if len(mats) > 1 else np.zeros(cells, np.int64))


def solve(ctx, insts, max_iter=500):
    """One batched solve of the instances; (x, iterations, residual norm, status) of each."""
    from gbfe import api

    off = np.concatenate([[0], np.cumsum([p["N"] for p in insts])]).astype(np.uint64)
    nd = np.concatenate([p["nd"] for p in insts])
    ids = np.concatenate([p["ids"].astype(np.int64) + int(o) for p, o in zip(insts, off)]).astype(np.uint32)
    mats, c2m, rows = [], [], []  # rows: (id, columns, weights)
    for p, o in zip(insts, off):
        c2m.append(p["c2m"] + len(mats))
        mats += p["mats"]
        rows += [(int(r) + int(o), (), ()) for r in p["rows"]]
        if p["hang"]:
            r, cols, w = p["hang"]
            rows.append((r + int(o), tuple(c + int(o) for c in cols), w))
    rows.sort()
    sizes = np.array([len(r[1]) for r in rows], np.uint32)
    cons = M.Constraints(np.array([r[0] for r in rows], np.uint32), sizes,
                         np.array([c for r in rows for c in r[1]], np.uint32),
                         (np.cumsum(sizes) - sizes).astype(np.uint32), np.array([w for r in rows for w in r[2]], float),
                         np.zeros(len(rows)))
    N = int(off[-1])
    basis = api.FEBasisManager(ctx, nd, ids, N, cons)
    K = api.IndexedCellMatrixOperatorContext(basis, np.concatenate(mats), np.concatenate(c2m).astype(np.uint32))
    J = api.PreconditionerJacobi(basis, np.concatenate([p["diag"] for p in insts]))
    b = api.MultiVector(basis, 1, init=np.concatenate([p["b"] for p in insts])[:, None])
    x = api.MultiVector(basis, 1)
    its, status, rn = api.pcg_solve_batched(K, J, b, x, off, max_iter, 1e-14, 1e-10, 1e10)
    ctx.check_status()
    xs = x.numpy()[:, 0]
    return [(xs[int(off[i]):int(off[i + 1])], int(its[i]), float(rn[i]), int(status[i])) for i in range(len(insts))]


@pytest.fixture(scope="module")
def alone(gpu_ctx):
    insts = instances()
    entries = [int((p["nd"].astype(np.int64) ** 2).sum()) for p in insts]
    assert min(entries) < LINE < max(entries)
    return insts, [solve(gpu_ctx, [p])[0] for p in insts]


def same(got, ref):
    assert got[1:] == ref[1:] and ref[3] == 0
    assert np.array_equal(got[0], ref[0])


@pytest.mark.parametrize("order", ["as given", "reversed", "only small", "only large"])
def test_results_do_not_depend_on_the_batch(gpu_ctx, alone, order):
    insts, ref = alone
    entries = np.array([int((p["nd"].astype(np.int64) ** 2).sum()) for p in insts])
    pick = {"as given": np.arange(len(insts)), "reversed": np.arange(len(insts))[::-1],
            "only small": np.flatnonzero(entries < LINE), "only large": np.flatnonzero(entries >= LINE)}[order]
    for k, got in zip(pick, solve(gpu_ctx, [insts[k] for k in pick])):
        same(got, ref[k])


@pytest.mark.parametrize("kind", ["hanging row", "own matrices", "large cells"])
@pytest.mark.parametrize("first", [False, True])
def test_results_do_not_depend_on_the_neighbour(gpu_ctx, alone, kind, first):
    insts, ref = alone
    extra = neighbour(kind, insts, np.random.default_rng(7))
    got = solve(gpu_ctx, [extra] + insts if first else insts + [extra])
    for g, r in zip(got[1:] if first else got[:-1], ref):
        same(g, r)


def test_neighbour_alone_and_in_the_batch(gpu_ctx, alone):
    """The neighbours' own results too (FMA products beside the tensor cores')."""
    insts, _ = alone
    for kind in ("own matrices", "large cells"):
        extra = neighbour(kind, insts, np.random.default_rng(7))
        same(solve(gpu_ctx, insts + [extra])[-1], solve(gpu_ctx, [extra])[0])
