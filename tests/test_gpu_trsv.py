"""Triangular solves: block chain, its correction, and the outer blocks for many right-hand
sides, at the edges of blocks and right-hand-side groups, both precisions."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 3, 4, 5, 7, 8, 9, 33])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 256, 511, 513, 1030])
def test_against_the_residual(ctx, n, nrhs):
    """Every right-hand side solved to the random-rounding estimate of its backward error
    (complex128: 4 sqrt(n) units) and, refined from complex64, to the acceptance 1e-13."""
    rng = np.random.default_rng(1000 * n + nrhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    norm = np.abs(A).sum(axis=1).max()
    for precision, bound in (("double", 4 * np.sqrt(n) * 2.0 ** -53 + 2.0 ** -53),
                             ("mixed", 1e-13)):
        X, _ = bemgpu.dense_solve(A, B, precision=precision, ctx=ctx)
        r = np.abs(B - A @ X).max(axis=0)
        scale = norm * np.abs(X).max(axis=0) + np.abs(B).max(axis=0)
        # numpy's own rounding of the residual adds sqrt(n) units
        assert np.all(r <= (bound + np.sqrt(n) * 2.0 ** -53) * scale), precision
