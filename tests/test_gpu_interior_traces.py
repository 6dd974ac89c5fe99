"""Interior field of a fluid body with its traces formed once (256 points or more) and where they
are used (fewer)."""
import numpy as np
import pytest

import bemgpu
from bemgpu import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["interior", "total"])
@pytest.mark.parametrize("count", [255, 256, 300])
def test_points_at_once_and_in_parts(ctx, count, field):
    """The same sums of 320 panels term by term: equal to the rounding of their trace products
    (a few units each, 320 of them, against the largest value)."""
    surf = bemgpu.mesh(*meshes.icosphere(0.01, 2))
    sol = bemgpu.bem(surf, bemgpu.FluidFilled(1.0357, 1.0279), 162.0, ctx=ctx)
    rng = np.random.default_rng(count)
    pts = rng.standard_normal((count, 3))
    pts *= (0.008 * rng.uniform(0.1, 1.0, count) / np.linalg.norm(pts, axis=1))[:, None]
    got = bemgpu.pressure(sol, pts, field=field)
    parts = np.concatenate([bemgpu.pressure(sol, pts[i:i + 100], field=field)
                            for i in range(0, count, 100)])
    assert np.max(np.abs(got - parts)) <= 320 * 4 * 2.0 ** -53 * np.max(np.abs(got))
    sol.close()
