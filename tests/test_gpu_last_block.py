"""Orders whose last outer block is short: its interchanges reach every earlier column (they
once covered the columns by count alone, and such complex64 factors were wrong enough to be
promoted)."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 130, 258, 270, 300, 385, 600, 1030, 2100])
def test_short_last_block(ctx, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    scale = np.abs(A).sum(axis=1).max()
    for precision in ("mixed", "double"):
        X, d = bemgpu.dense_solve(A, B, precision=precision, ctx=ctx)
        r = np.abs(B - A @ X).max()
        assert r <= 1e-13 * (scale * np.abs(X).max() + np.abs(B).max())
        if precision == "mixed":
            # condition numbers of a few thousand: far from the guard, and each step of the
            # refinement gains about three digits
            assert d["factor_precision"] == "single" and d["refinement_iterations"] <= 6
