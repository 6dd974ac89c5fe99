"""The complex128 LU: 32-column panels, 128-column blocks whose updates run on the tensor
cores from integer digits.  Orders at the edges of panels, blocks and tiles, against the
residual in numpy."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _matrix(kind, n, rng):
    if kind == "equal":          # constant entries: every digit product adds up coherently
        return np.full((n, n), 0.49999999, dtype=complex) + np.diag(np.linspace(1, 2, n))
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if kind == "graded":         # entries of one row differ by many powers of two
        A = A * 2.0 ** rng.integers(-40, 1, (n, n))
        A = A + np.diag(np.full(n, 4.0))
    if kind == "tiny":           # exponents near the lower end of the format
        A = A * 2.0 ** -900
    return A


@pytest.mark.parametrize("kind", ["normal", "equal", "graded", "tiny"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 160, 161, 256, 289, 513])
def test_backward_error(ctx, kind, n):
    """Normwise backward error of the solve within the random-rounding estimate 4 sqrt(n)
    of the unit roundoff (the n-term sums of the factorisation and of the two solves), not
    above twice the FP64 pipe's beyond one rounding."""
    rng = np.random.default_rng(n)
    A = _matrix(kind, n, rng)
    X = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    B = A @ X

    def backward(Y):
        r = np.abs(B - A @ Y).max(axis=0)
        return float((r / (np.abs(A).sum(axis=1).max() * np.abs(Y).max(axis=0))).max())

    Y, d = bemgpu.dense_solve(A, B, equilibrate=kind != "tiny", ctx=ctx)
    ctx.set_tensor_lu(False)
    try:
        Z, _ = bemgpu.dense_solve(A, B, equilibrate=kind != "tiny", ctx=ctx)
    finally:
        ctx.set_tensor_lu(True)
    assert d["factor_precision"] == "double"
    assert backward(Y) <= 4 * np.sqrt(n) * EPS + EPS
    assert backward(Y) <= 2 * backward(Z) + 4 * EPS
