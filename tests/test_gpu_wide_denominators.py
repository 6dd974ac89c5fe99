"""|A||x| of many right-hand sides: FP32 sums of at most 2048 columns."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu


def test_sums_of_many_columns(ctx):
    """One large term before 8191 terms below half a unit of its rounding: FP32 sums of 2048 columns
    are off by at most 2047 roundings of 2^-24, one sum of all of them loses 2.2e-4 of |b| + |A||x|."""
    n, nrhs = 8192, 16
    rng = np.random.default_rng(5)

    def phases(shape):
        t = rng.uniform(0, 2 * np.pi, shape)
        return np.cos(t) + 1j * np.sin(t)

    A = phases((n, n))
    A[np.arange(n), np.arange(n)] *= 1000.0  # well conditioned
    X = 2.3e-4 * phases((n, nrhs))
    X[0] = 4096.0 * phases(nrhs)
    B = A @ X
    # accepted after the complex64 solve, whose residual both sides know to six digits
    Y, d = bemgpu.dense_solve(A, B, precision="mixed", ctx=ctx,
                              refinement=dict(tolerance=1e-3, maxiter=10))
    r = np.abs(B - A @ Y)
    want = (r / (np.abs(A) @ np.abs(Y) + np.abs(B))).max()
    assert want > 1e-10
    assert abs(d["componentwise_backward_error"] / want - 1) <= 2047 * 2.0 ** -24 + 1e-5
