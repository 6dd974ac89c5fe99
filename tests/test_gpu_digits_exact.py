"""Digit products on the tensor cores with operands whose products and sums are exact in FP64:
factors, solutions and residuals come out exactly, so one lost, doubled or reordered
accumulation shows."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu

FILL = 4  # nonzero entries of a solution beside the first


def _fixed(rng, shape, bits):
    """Complex multiples of 2^-bits, parts below 1/2 in size."""
    v = rng.integers(-2 ** (bits - 1) + 1, 2 ** (bits - 1), shape + (2,)) * 2.0 ** -bits
    return v[..., 0] + 1j * v[..., 1]


def _system(rng, n, blocks, bits_n, bits_m):
    """[[I, M], [N, I + N M]] with 128 blocks leading rows: the factors are [[I, 0], [N, I]] and
    [[I, M], [0, I]], without interchanges as |re| + |im| < 1 in N.  Row and column 0 are e_0."""
    k = 128 * blocks
    N = _fixed(rng, (n - k, k), bits_n)
    M = _fixed(rng, (k, n - k), bits_m)
    N[:, 0] = 0
    M[0] = 0
    A = np.eye(n, dtype=complex)
    A[:k, k:] = M
    A[k:, :k] = N
    A[k:, k:] += N @ M
    return A


@pytest.mark.parametrize("nrhs", [3, 16, 37])
@pytest.mark.parametrize("bits", [(30, 8), (8, 30), (19, 19)])
@pytest.mark.parametrize("n,blocks", [(129, 1), (300, 1), (427, 2), (1884, 3)])
def test_factors_solutions_and_residuals_are_exact(ctx, n, blocks, bits, nrhs):
    """Every sum is of multiples of 2^-38 below 2^13: N M is at most 384 terms of size 1/2, a row
    of A X at most FILL entries of N M and the first unknown."""
    rng = np.random.default_rng(n + nrhs)
    A = _system(rng, n, blocks, *bits)
    X = np.zeros((n, nrhs), dtype=complex)
    for r in range(nrhs):
        at = rng.choice(np.arange(1, n), FILL, replace=False)
        X[at, r] = rng.choice([1, -1, 1j, -1j], FILL)
    X[0] = 2.0 ** 12  # the largest entry of b: right-hand sides are scaled by it, here exactly
    B = A @ X
    assert np.abs(B[1:]).max() < 2.0 ** 12 and sum(bits) + 13 <= 53
    Y, d = bemgpu.dense_solve(A, B, equilibrate=False, ctx=ctx)
    assert d["factor_precision"] == "double"
    assert np.array_equal(Y, X)
    assert d["relative_residual"] == 0.0
