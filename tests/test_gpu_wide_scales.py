"""Products of one system with many right-hand sides where the unknowns differ in size: by column
scales, inside a vector, and between the pressures and fluxes of a fluid body.  The digit
products' exponents are shared by a row and 128 columns, so their error must not become one of
the residual."""
import math

import numpy as np
import pytest

import bemgpu
from bemgpu import meshes

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
# share of |A||x| by which a product may be off: E <= 64 |A||x| of the error bound's unit
# 2^-56 E, entries of mixed signs at 8 units
SHARE = 64 * 8 * 2.0 ** -56


def _residual(A, X, B):
    """B - A X in extended precision, and |A||X|."""
    ar, ai, xr, xi = (v.astype(np.longdouble) for v in (A.real, A.imag, X.real, X.imag))
    r = B.real - (ar @ xr - ai @ xi) + 1j * (B.imag - (ar @ xi + ai @ xr))
    return np.asarray(r, dtype=complex), np.abs(A) @ np.abs(X)


def _check(ctx, A, B, precision):
    X, d = bemgpu.dense_solve(A, B, precision=precision, ctx=ctx)
    n = len(A)
    R, AX = _residual(A, X, B)
    den = AX + np.abs(B)
    if precision == "mixed":  # accepted at 1e-13 of den, as the products saw it
        assert np.all(np.abs(R) <= (1e-13 * (1 + 1e-3) + SHARE) * den)
    off = SHARE + 2 * n * U  # of the reported residual: the product's error and its rounding
    norm = np.linalg.norm(B, axis=0)
    true = (np.linalg.norm(R, axis=0) / norm).max()
    slack = off * (np.linalg.norm(den, axis=0) / norm).max()
    assert abs(d["relative_residual"] - true) <= slack
    comp = (np.abs(R) / den).max()
    assert abs(d["componentwise_backward_error"] - comp) <= off + 1e-3 * comp


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("nrhs", [15, 16, 33])
@pytest.mark.parametrize("n", [129, 200])
@pytest.mark.parametrize("scale", [3, 6, 8])
def test_columns_of_different_sizes(ctx, scale, n, nrhs, precision):
    rng = np.random.default_rng(n + nrhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.eye(n)
    A = A * 10.0 ** rng.uniform(-scale, scale, n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    _check(ctx, A, B, precision)


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("n,nrhs", [(200, 200), (700, 16), (700, 40)])
def test_vectors_of_different_sizes(ctx, n, nrhs, precision):
    """The inverse's columns of a matrix near the identity: their entries spread over 1e-5, which
    no common scale of the unknowns takes out.  Few columns: some entries of the product are
    formed again; all of them: the whole product is."""
    rng = np.random.default_rng(n + nrhs)
    A = np.eye(n) + 1e-5 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    _check(ctx, A, np.eye(n, dtype=complex)[:, :nrhs], precision)


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("level", [2, None])
def test_fluid_of_a_small_body_at_a_high_frequency(ctx, level, precision):
    """Pressures of size 1 beside fluxes of size k = 10^4 in one block of 128 unknowns (320 and 252
    panels): every angle converges to its own solve, both with backward errors below 1e-13 (mixed)
    of systems with condition numbers below 1e3."""
    k = 1e4
    nodes, tris = (meshes.icosphere(0.01, level) if level else
                   meshes.uv_spheroid(0.02, 0.01, 14, 10, jitter=0.02, seed=3))
    surf = bemgpu.mesh(nodes * (159.0 / k), tris)
    f = bemgpu.Factor(surf, bemgpu.FluidFilled(1.2, 1.1), k, ctx=ctx, precision=precision)
    angles = np.linspace(0.1, 3.0, 16)
    many = f.solve(angles, 0.3)
    d = many.diagnostics()
    assert d["factor_precision"] == ("single" if precision == "mixed" else "double")
    assert d["componentwise_backward_error"] <= 1e-13
    for r in (0, 7, 15):
        one = f.solve([angles[r]], 0.3)
        for a, b in zip(many.traces(r), one.traces(0)):
            assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b)
        one.close()
    many.close()
    f.close()
