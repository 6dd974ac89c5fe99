"""The complex128 LU without equilibration: rows and columns of very different sizes, against the
FP64 pipe's factorisation entry by entry."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _componentwise(A, Y, B):
    """Largest |B - A Y| / (|A||Y| + |B|), the residual in extended precision."""
    ar, ai, xr, xi = (v.astype(np.longdouble) for v in (A.real, A.imag, Y.real, Y.imag))
    r = np.hypot((B.real - (ar @ xr - ai @ xi)).astype(float),
                 (B.imag - (ar @ xi + ai @ xr)).astype(float))
    return (r / (np.abs(A) @ np.abs(Y) + np.abs(B))).max()


@pytest.mark.parametrize("scale", [4, 8])
@pytest.mark.parametrize("which", ["rows", "columns", "both"])
@pytest.mark.parametrize("n", [129, 256, 385, 513])
def test_componentwise_backward_error(ctx, which, scale, n):
    """Not above twice the FP64 pipe's beyond its own rounding, as for equilibrated systems: the
    digits that are dropped are below the rounding errors of the sums."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if which != "columns":
        A = A * 10.0 ** rng.uniform(-scale, scale, n)[:, None]
    if which != "rows":
        A = A * 10.0 ** rng.uniform(-scale, scale, n)
    B = A @ (rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3)))
    Y, _ = bemgpu.dense_solve(A, B, equilibrate=False, ctx=ctx)
    ctx.set_tensor_lu(False)
    try:
        Z, _ = bemgpu.dense_solve(A, B, equilibrate=False, ctx=ctx)
    finally:
        ctx.set_tensor_lu(True)
    assert _componentwise(A, Y, B) <= 2 * _componentwise(A, Z, B) + 4 * EPS
