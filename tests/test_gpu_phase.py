"""FP64 quadrature phases: short, middle and long panels against the oracle's operators, and the
pressure's region test near the surface."""
import math

import numpy as np
import pytest

import bemgpu
from bemgpu import meshes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge_k", [0.05, 0.52, 0.54, 1.59, 1.61, 4.0])
def test_operators_on_both_sides_of_the_phase_rules(ctx, edge_k):
    """Elementwise to 1e-12 of the largest entry, the tolerance of the FP64 operators."""
    nodes, tris = meshes.uv_spheroid(1.0, 0.6, 12, 9, jitter=0.02, seed=4)
    P = O.Panels(nodes, tris)
    k = edge_k / float(P.diams.max())
    for bc, ref in ((bemgpu.Rigid(), O.assemble_bm(P, k)),
                    (bemgpu.FluidFilled(1.2, 1.1), (O.assemble_fluid(P, k, 1.2, 1.1),))):
        got = bemgpu.assemble(bemgpu.mesh(nodes, tris), bc, k, ctx=ctx)
        got = got if isinstance(got, tuple) else (got,)
        for g, r in zip(got, ref):
            assert np.max(np.abs(g - r)) <= 1e-12 * np.max(np.abs(r))


@pytest.mark.parametrize("edge_k", [0.3, 1.0, 3.0])
def test_far_field_phase_series(ctx, edge_k):
    """One and many directions (both kernels) against the oracle's sum."""
    nodes, tris = meshes.uv_spheroid(1.0, 0.6, 12, 9, jitter=0.02, seed=5)
    P = O.Panels(nodes, tris)
    k = edge_k / float(P.diams.max())
    sol = bemgpu.bem(bemgpu.mesh(nodes, tris), bemgpu.Rigid(), k, ctx=ctx)
    p, q = sol.traces()
    rng = np.random.default_rng(1)
    d = rng.normal(size=(130, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    want = np.array([O.far_field(P, k, x, p, q) for x in d])
    scale = np.max(np.abs(want))
    for n in (1, 31, 32, 130):
        assert np.max(np.abs(sol.far_field(d[:n]) - want[:n])) <= 1e-12 * scale


def test_region_of_points_close_to_the_surface(ctx):
    """Points a hair inside and outside every kind of place of a panel get their own side's
    field, as the oracle's FP64 solid angle decides."""
    nodes, tris = meshes.icosphere(1.0, 2)
    surf = bemgpu.mesh(nodes, tris)
    bc = bemgpu.FluidFilled(1.2, 1.1)
    sol = bemgpu.bem(surf, bc, 1.3, incidence_angle=math.pi / 3, incidence_azimuth=0.4, ctx=ctx)
    P = O.Panels(nodes, tris)
    p, q = sol.traces()
    d = O.incidence_direction(math.pi / 3, 0.4)
    pts = []
    for t in (0, 57, 211):
        for bary in ((1 / 3, 1 / 3, 1 / 3), (0.98, 0.01, 0.01), (0.5, 0.499, 0.001)):
            x = np.asarray(bary) @ P.vertices[t]
            for h in (1e-9, 1e-6, 1e-3):
                pts += [x + h * P.normals[t], x - h * P.normals[t]]
    pts = np.array(pts)
    got = bemgpu.pressure(sol, pts)
    want = O.pressure(P, 1.3, pts, p, q, d, field="total", g=1.2, h=1.1, fluid=True)
    assert np.max(np.abs(got - want)) <= 1e-8 * np.max(np.abs(want))
