"""Row-wise products of more right-hand sides than one launch's grid holds (2047 groups of four,
with 32 column chunks each)."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [8188, 8189, 9001])
def test_row_wise_products(ctx, nrhs):
    """Solved to the backward error of an FP64 factorisation (4 sqrt(n) units), with a reported
    residual that the row-wise products formed for every right-hand side."""
    n = 33
    rng = np.random.default_rng(nrhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    ctx.set_tensor_lu(False)
    try:
        X, d = bemgpu.dense_solve(A, B, ctx=ctx)
    finally:
        ctx.set_tensor_lu(True)
    eps = 2.0 ** -53
    r = np.abs(B - A @ X).max(axis=0)
    scale = np.abs(A).sum(axis=1).max() * np.abs(X).max(axis=0) + np.abs(B).max(axis=0)
    assert np.all(r <= (5 * np.sqrt(n) + 1) * eps * scale)
    assert 0.0 < d["normwise_backward_error"] <= (5 * np.sqrt(n) + 1) * eps
