"""Row-wise sweeps, statistics and row permutations around a solve, at the edges of their splits
(column chunks by order, statistics by 256 rows, pivots by tiles of 2048), with rows of very
different sizes."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17, 255, 511, 512, 513, 2047, 2049, 2560, 2561, 4096, 5121])
def test_rows_of_different_sizes(ctx, n):
    """Mixed, promoted to complex128 or not: every row of the residual within the acceptance (1e-13
    of |b| + |A||x|, and numpy's own rounding of the row).  Double: each row to 1e-13 of its norm times max |x|."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    size = 10.0 ** rng.uniform(-12, 12, n)
    A *= size[:, None]
    B *= size[:, None]
    own = np.sqrt(n) * 2.0 ** -52
    for precision in ("mixed", "double"):
        X, _ = bemgpu.dense_solve(A, B, precision=precision, ctx=ctx)
        r = np.abs(B - A @ X)
        if precision == "mixed":
            assert np.all(r <= (1e-13 + own) * (np.abs(A) @ np.abs(X) + np.abs(B)))
        else:
            rows = np.abs(A).sum(axis=1)[:, None]
            assert np.all(r <= (1e-13 + own) * (rows * np.abs(X).max(axis=0) + np.abs(B)))
