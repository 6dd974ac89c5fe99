"""Every launch shape of the panel factorisation gives the same bits: clusters of 1 to 16 CTAs with
1 to 10 rows per thread in registers, and the kernel that streams panels beyond that."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu


def _factors(A, out, piv):
    """Residual |P A - L U| relative to |L||U|, entry by entry."""
    n, nb = A.shape
    P = A.copy()
    for c, p in enumerate(piv):
        P[[c, p]] = P[[p, c]]
    L = np.tril(out, -1)
    L[np.arange(nb), np.arange(nb)] = 1.0
    U = np.triu(out[:nb])
    return (np.abs(P - L @ U) / (np.abs(L) @ np.abs(U))).max()


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("n", [32, 33, 100, 513, 1030, 2700, 5200, 11000])
def test_same_bits_in_every_shape(ctx, n, precision):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, 32)) + 1j * rng.standard_normal((n, 32))
    if precision == "mixed":
        A = A.astype(np.complex64).astype(complex)
    A[n // 2, 3] = 0
    out, piv = ctx.debug_panel(A, precision)
    # 32 products and sums per entry
    eps = 2.0 ** -24 if precision == "mixed" else 2.0 ** -53
    assert _factors(A, out, piv) <= 2 * 32 * eps
    for cluster in (1, 2, 4, 8, 16):
        for streaming in (False, True):
            o, p = ctx.debug_panel(A, precision, cluster, streaming)
            assert np.array_equal(p, piv) and np.array_equal(o, out), (cluster, streaming)


@pytest.mark.parametrize("precision", ["mixed", "double"])
def test_columns_of_zeros_and_ties(ctx, precision):
    """A zero column (no interchange) and entries of equal size (the first row wins)."""
    rng = np.random.default_rng(1)
    A = rng.choice([1.0, -1.0], (300, 32)) + 0j
    A[:, 5] = 0
    out, piv = ctx.debug_panel(A, precision)
    assert piv[0] == 0 and piv[5] == 5
    for cluster in (1, 4, 16):
        for streaming in (False, True):
            o, p = ctx.debug_panel(A, precision, cluster, streaming)
            assert np.array_equal(p, piv) and np.array_equal(o, out), (cluster, streaming)
