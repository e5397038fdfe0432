"""m x m eigenproblem above the host's range (FP32 decomposition refined to FP64): Rayleigh-Ritz in an invariant
subspace of a block-diagonal operator whose eigenvalues are chosen, so that the projected matrix is dense with that
spectrum.

Bound, for eigenvalues, residual and orthogonality alike, relative to the largest eigenvalue of the operator:
4 m 2^-52 (each entry of the projected matrix and of the rotated vectors is a sum of m or 64 rounded products)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ND = 64


def rayleigh_ritz(ctx, w, seed=0):
    from gbfe import api

    m = w.size
    rng = np.random.default_rng(seed)
    cells = m // ND + 1
    N = cells * ND
    w_all = np.concatenate([w, np.abs(w).max() * rng.random(N - m)])
    V = [np.linalg.qr(rng.standard_normal((ND, ND)))[0] for _ in range(cells)]
    mats = np.stack([(v * w_all[c * ND:(c + 1) * ND]) @ v.T for c, v in enumerate(V)])
    mats = (mats + mats.transpose(0, 2, 1)) / 2
    Vm = np.zeros((N, N))
    for c, v in enumerate(V):
        Vm[c * ND:(c + 1) * ND, c * ND:(c + 1) * ND] = v
    X0 = Vm[:, :m] @ np.linalg.qr(rng.standard_normal((m, m)))[0]
    basis = api.FEBasisManager(ctx, np.full(cells, ND, np.uint32), np.arange(N, dtype=np.uint32), N)
    H = api.KohnShamOperatorContextFE(basis, mats.ravel())
    X, Y = api.MultiVector(basis, m, init=X0), api.MultiVector(basis, m)
    eig = np.asarray(api.RayleighRitzEigenSolver.solve(H, X, Y))
    Z = Y.numpy()
    HZ = np.concatenate([mats[c] @ Z[c * ND:(c + 1) * ND] for c in range(cells)])
    return eig, Z, HZ


def spectrum(kind, m, rng):
    if kind == "separate":
        return rng.standard_normal(m)
    if kind == "even":
        return np.linspace(-1.0, 1.0, m)
    if kind == "triples":
        return np.repeat(np.linspace(-1.0, 1.0, m // 3 + 1), 3)[:m]
    if kind == "pairs apart by 1e-6":
        return (np.repeat(rng.random(m // 2 + 1), 2) + 1e-6 * (np.arange(2 * (m // 2 + 1)) % 2))[:m]
    if kind.startswith("cluster"):  # "cluster k": k eigenvalues within 1e-8
        k = int(kind.split()[1])
        return np.concatenate([0.5 + 1e-8 * rng.random(k), np.linspace(1.0, 2.0, m - k)])
    if kind == "graded":
        return 10.0 ** np.linspace(-12, 0, m)
    if kind == "equal":
        return np.full(m, 0.75)
    raise ValueError(kind)


@pytest.mark.parametrize("m,kind,scale", [
    (129, "separate", 1.0), (144, "separate", 1.0), (255, "separate", 1.0), (256, "separate", 1.0),
    (257, "separate", 1.0), (512, "separate", 1.0), (768, "separate", 1.0), (769, "separate", 1.0),
    (256, "even", 1.0), (192, "triples", 1.0),
    (160, "pairs apart by 1e-6", 1.0), (160, "cluster 2", 1.0), (160, "cluster 63", 1.0), (160, "cluster 64", 1.0),
    (160, "cluster 65", 1.0), (160, "graded", 1.0), (160, "equal", 1.0), (160, "separate", 1e60),
    (160, "triples", 1e-60)])
def test_chosen_spectrum(gpu_ctx, m, kind, scale):
    w = scale * spectrum(kind, m, np.random.default_rng(m))
    eig, Z, HZ = rayleigh_ritz(gpu_ctx, w, seed=m)
    tol = 4 * m * 2.0 ** -52
    top = np.abs(w).max()
    assert np.abs(eig - np.sort(w)).max() <= tol * top
    assert np.abs(Z.T @ Z - np.eye(m)).max() <= tol
    assert np.abs(HZ - Z * eig).max() <= tol * top
