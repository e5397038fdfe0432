"""FP64-accurate sliced cell product with the digits of both operands at their limits.

Operands of five digits near 127 (or -128) each: the kept products (slices s + t <= 8) fill the levels as far as they
can be filled over up to 256 rows, level 6 past 2^24.  Every accumulator has to hold its sum exactly, so the result is
the sum of the kept products rounded once: the same double as integer arithmetic gives."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLICES = 5


def operand(shape, sign, rng):
    """Values 2 sum_s d_s 256^-s in (0.5, 1) or (-1, -0.5), and their digits."""
    d = sign * rng.integers(120, 128, (SLICES,) + shape)
    d[1:] -= sign < 0  # (-128 .. -121 below the first, which stays above -128: |v| < 1)
    fixed = sum(d[s].astype(np.int64) * 256 ** (SLICES - 1 - s) for s in range(SLICES))
    return np.ldexp(fixed.astype(np.float64), 1 - 8 * SLICES), d.astype(np.int64)


@pytest.mark.parametrize("nd", [64, 128, 146, 147, 204, 205, 216, 255, 256])
@pytest.mark.parametrize("sign", [1, -1])
def test_kept_products_are_rounded_once(gpu_ctx, nd, sign):
    from gbfe import api

    m, rng = 70, np.random.default_rng(nd)
    A, ad = operand((nd, nd), sign, rng)
    X0, xd = operand((nd, m), 1, rng)
    assert 0.5 < np.abs(A).min() and np.abs(A).max() < 1.0 and np.abs(X0).max() < 1.0
    kept = np.zeros((nd, m), dtype=object)
    for s in range(1, SLICES + 1):
        for t in range(1, SLICES + 1):
            if s + t <= 8:
                kept += (ad[s - 1] @ xd[t - 1]).astype(object) * 256 ** (8 - s - t)
    if nd == 256:
        level6 = sum(ad[s - 1] @ xd[5 - s] for s in range(1, 6))
        assert np.abs(level6).max() > 2 ** 24
    exact = np.array([[float(Fraction(int(k) * 4, 256 ** 8)) for k in row] for row in kept])
    basis = api.FEBasisManager(gpu_ctx, np.array([nd], np.uint32), np.arange(nd, dtype=np.uint32), nd)
    H = api.KohnShamOperatorContextFE(basis, A.ravel(), fp64_tensor=True)
    gpu_ctx.set_fp64_apply(1)
    try:
        Y = api.MultiVector(basis, m)
        H.apply(api.MultiVector(basis, m, init=X0), Y)
        got = Y.numpy()
    finally:
        gpu_ctx.set_fp64_apply(0)
    gpu_ctx.check_status()
    assert np.array_equal(got, exact), np.abs(got - exact).max() / np.spacing(np.abs(exact).max())
