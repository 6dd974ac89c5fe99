"""The panel factorisation holds rows in registers: its pivots and factors must not depend on
the cluster size, the rows per thread or the batch it runs in."""
import math

import numpy as np
import pytest

import bemgpu
from bemgpu import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("count", [1, 5, 20, 80])
def test_same_in_every_batch_size(ctx, precision, count):
    """One body alone and among others (clusters of 16 down to one CTA per system): the same
    bits."""
    surf = bemgpu.mesh(*meshes.icosphere(0.01, 2))
    other = bemgpu.mesh(*meshes.uv_spheroid(0.02, 0.01, 12, 9, jitter=0.02, seed=2))
    k = 2 * math.pi * 38e3 / 1477.4

    def solve(items):
        fs = bemgpu.factor_batch([(s, bemgpu.Rigid(), kk, dict(precision=precision))
                                  for s, kk in items], ctx=ctx)
        sols = bemgpu.solve_batch(fs, [[0.7]] * len(fs))
        out = sols[0].traces()[0], sols[0].far_field()[0]
        for x in sols + fs:
            x.close()
        return out

    alone = solve([(surf, k)])
    mixed = solve([(surf, k)] + [(other, k * (1 + 0.01 * i)) for i in range(count - 1)])
    assert np.array_equal(alone[0], mixed[0]) and alone[1] == mixed[1]


@pytest.mark.parametrize("n", [33, 520, 2600, 9000])
def test_pivots_of_a_shifted_permutation(ctx, n):
    """A permuted diagonal with tiny fill: every pivot is the single large entry of its
    column, wherever its row lives (all rows-per-thread variants), ties excluded."""
    rng = np.random.default_rng(n)
    perm = rng.permutation(n)
    A = np.zeros((n, n), dtype=np.complex128)
    A[perm, np.arange(n)] = 1.0 + rng.uniform(0.0, 1.0, n)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    y, _ = bemgpu.dense_solve(A, A @ x, ctx=ctx)
    # one product and one quotient per entry: a few units of the rounding error
    assert np.max(np.abs(y - x) / np.abs(x)) <= 8 * 2.0 ** -53
    y, d = bemgpu.dense_solve(A, A @ x, precision="mixed", ctx=ctx)
    # the refinement's acceptance (componentwise backward error 1e-13), doubled for the
    # rounding of A @ x: on a diagonal that is the relative error of every entry
    assert d["factor_precision"] == "single"
    assert np.max(np.abs(y - x) / np.abs(x)) <= 2e-13
