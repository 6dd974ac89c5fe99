"""The pressure's region test for bodies whose extent FP32 products of three distances do not
hold: the same fields as those of a unit body at the same k a."""
import numpy as np
import pytest

import bemgpu
from bemgpu import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1e-16, 1e-14, 1e-11, 1e11, 1e14])
def test_fields_scale_with_the_body(ctx, size):
    """Inside and outside of a fluid sphere, well off its surface; the solutions differ by the
    rounding of the scaled coordinates."""
    nodes, tris = meshes.icosphere(1.0, 2)
    rng = np.random.default_rng(1)
    d = rng.normal(size=(40, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    pts = d * np.where(np.arange(40) % 2, rng.uniform(0.05, 0.7, 40),
                       rng.uniform(1.4, 3.0, 40))[:, None]
    bc, angle = bemgpu.FluidFilled(1.2, 1.1), 0.7
    unit = bemgpu.bem(bemgpu.mesh(nodes, tris), bc, 1.3, incidence_angle=angle, ctx=ctx)
    sol = bemgpu.bem(bemgpu.mesh(nodes * size, tris), bc, 1.3 / size, incidence_angle=angle,
                     ctx=ctx)
    want = bemgpu.pressure(unit, pts)
    got = bemgpu.pressure(sol, pts * size)
    assert np.max(np.abs(got - want)) <= 1e-9 * np.max(np.abs(want))
