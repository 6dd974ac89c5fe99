"""Products of many right-hand sides when memory is short: the slices are taken if there is room,
and the row-wise products need none."""
import numpy as np
import pytest

import bemgpu

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _solve(budget, A, B, tensor):
    c = bemgpu.Context(0, hbm_budget_bytes=budget)
    try:
        c.set_tensor_lu(tensor)
        return bemgpu.dense_solve(A, B, ctx=c)
    except bemgpu.BEMGPUError as e:
        assert "budget" in str(e)
        return None
    finally:
        c.close()


def test_least_budget_is_that_of_the_row_wise_products(ctx):
    n, nrhs = 300, 400
    rng = np.random.default_rng(3)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    lo, hi = 1, 512  # MB: too little, enough
    assert _solve(lo * MB, A, B, False) is None and _solve(hi * MB, A, B, False) is not None
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if _solve(mid * MB, A, B, False) is None:
            lo = mid
        else:
            hi = mid
    eps = 2.0 ** -53
    for budget in (hi, hi + 4, hi + 8, 512):  # no panel, one, a few, all
        got = _solve(budget * MB, A, B, True)
        assert got is not None, budget
        X, d = got
        r = np.abs(B - A @ X).max(axis=0)
        scale = np.abs(A).sum(axis=1).max() * np.abs(X).max(axis=0) + np.abs(B).max(axis=0)
        assert np.all(r <= (5 * np.sqrt(n) + 1) * eps * scale)
        assert d["normwise_backward_error"] <= (5 * np.sqrt(n) + 1) * eps


def test_least_budget_of_a_double_factorisation(ctx):
    """The slices of its updates are taken if there is room: the least budget is that of the FP64
    pipe and the descriptors."""
    n = 900
    rng = np.random.default_rng(5)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    lo, hi = 1, 512
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if _solve(mid * MB, A, B, False) is None:
            lo = mid
        else:
            hi = mid
    eps = 2.0 ** -53
    for budget in (hi + 1, 512):
        got = _solve(budget * MB, A, B, True)
        assert got is not None, budget
        r = np.abs(B - A @ got[0]).max(axis=0)
        scale = np.abs(A).sum(axis=1).max() * np.abs(got[0]).max(axis=0) + np.abs(B).max(axis=0)
        assert np.all(r <= (5 * np.sqrt(n) + 1) * eps * scale)


def test_partial_sums_of_many_right_hand_sides(ctx):
    """Eight chunks of partial sums per right-hand side (of 24 bytes an unknown), the seven other
    vectors and the few MB of a system of 300 unknowns are enough."""
    n, nrhs = 300, 400
    rng = np.random.default_rng(4)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    need = n * nrhs * (8 * 24 + 7 * 16) + 16 * MB
    assert _solve(need, A, B, True) is not None


def test_server_under_a_budget_with_many_angles(ctx):
    """Requests whose slices count in the admission: all complete, none runs out of memory."""
    from bemgpu import meshes
    c = bemgpu.Context(0, hbm_budget_bytes=120 * MB)
    surf = bemgpu.mesh(*meshes.uv_spheroid(0.02, 0.008, 24, 16, jitter=0.02, seed=5))
    srv = bemgpu.Server(c, max_batch=8)
    try:
        angles = np.linspace(0.1, 3.0, 24)
        tickets = [srv.submit(surf, bemgpu.Rigid(), [250.0 + 10 * i], angles, precision="mixed")
                   for i in range(6)]
        res = [srv.wait(t)[0] for t in tickets]
        st = srv.stats()
    finally:
        srv.close()
        c.close()
    assert st["completed"] == 6 and st["failed"] == 0
    assert all(np.all(np.isfinite(r)) for r in res)
