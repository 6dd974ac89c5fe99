"""Products of one system with many right-hand sides (digit slices on the tensor cores): a
sweep of many angles gives the single solves, on both sides of the right-hand-side rule."""
import math

import numpy as np
import pytest

import bemgpu
from bemgpu import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("boundary", [bemgpu.Rigid(), bemgpu.PressureRelease(),
                                      bemgpu.FluidFilled(1.2, 1.1)])
@pytest.mark.parametrize("count", [15, 16, 33])
def test_sweep_is_the_single_solves(ctx, boundary, precision, count):
    """Traces of every angle against its own solve.  Both are solutions to a backward error
    below 1e-13 (mixed) of systems with condition numbers below 1e3."""
    surf = bemgpu.mesh(*meshes.uv_spheroid(0.02, 0.01, 14, 10, jitter=0.02, seed=3))
    k = 2 * math.pi * 38e3 / 1500.0
    angles = np.linspace(0.1, 3.0, count)
    f = bemgpu.Factor(surf, boundary, k, ctx=ctx, precision=precision)
    many = f.solve(angles, 0.3)
    for r in (0, count // 2, count - 1):
        one = f.solve([angles[r]], 0.3)
        for a, b in zip(many.traces(r), one.traces(0)):
            assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b)
    d = many.diagnostics()
    assert d["relative_residual"] <= 1e-12
