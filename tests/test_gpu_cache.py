"""Device memory kept between calls: calls of one shape reuse it, gbfe_ctx_release_cache gives it back, and results do
not depend on it."""
import numpy as np
import pytest

import gbfe.mesh as M

pytestmark = pytest.mark.gpu


def test_kept_memory_is_bounded_and_given_back(gpu_ctx):
    import torch
    from gbfe import api

    p = M.build_problem(8, 3, 16.0, np.zeros((0, 3)), np.zeros(0), 0.5, matrices=())
    basis = api.FEBasisManager.from_problem(gpu_ctx, p)
    X = api.MultiVector(basis, 256, init=M.random_block(p.n_dofs, 256, 1))
    Y = api.MultiVector(basis, 256)
    T = M.random_block(256, 256, 2)

    def call():
        api.rotate(X, T, Y)
        return api.gram(X, Y)

    first = call()
    gpu_ctx.release_cache()
    gpu_ctx.synchronize()
    base = torch.cuda.mem_get_info(0)[0]
    call()
    kept = base - torch.cuda.mem_get_info(0)[0]
    for _ in range(4):
        assert np.array_equal(call(), first)
    assert base - torch.cuda.mem_get_info(0)[0] == kept
    assert 0 <= kept <= 4 << 30
    gpu_ctx.release_cache()
    assert torch.cuda.mem_get_info(0)[0] >= base
    assert np.array_equal(call(), first)
