"""Lanczos bounds of an operator whose Krylov space is one vector: the first step is the last one read, whatever number
was asked for, and the steps after it are not queued on and on (about seven launches each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [2, 63, 64, 65, 3000])
def test_breakdown_ends_the_steps(gpu_ctx, steps):
    from gbfe import api

    nd, cells = 27, 8
    N = nd * cells
    basis = api.FEBasisManager(gpu_ctx, np.full(cells, nd, np.uint32), np.arange(N, dtype=np.uint32), N)
    H = api.KohnShamOperatorContextFE(basis, np.tile(2.0 * np.eye(nd).ravel(), cells))
    Mo = api.CFEOverlapOperatorContext(basis, np.tile(np.eye(nd).ravel(), cells))
    Mi = api.CFEOverlapInverseOpContextGLL(basis, np.ones(N))
    before = gpu_ctx.kernel_launches()
    lo, hi, beta = api.lanczos_bounds(H, Mo, Mi, steps=steps)
    # alpha = q . 2 q with |q| = 1: N products, two roundings of the norm
    assert abs(lo - 2.0) <= N * 2.0 ** -52 and hi == lo and beta < 1e-14
    assert gpu_ctx.kernel_launches() - before <= 10 * min(steps, 64) + 10
    gpu_ctx.check_status()
