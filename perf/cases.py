"""The workloads whose times are followed: the framework's public calls over the range of
sizes, boundary conditions, precisions and options that its users have.

A case is one call (or one short sequence of calls) of the Python package, on surfaces that
the caller already holds.  `listed()` names the fixed cases, `draw(rng)` gives further ones
from the same ranges.  `exact()` restates the discretisation in 64-bit torch operations:
constant panels collocated at their centroids with closed-form near terms, and the Nyström
nodes with the plane-wave density interpolation.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "acousticscattering.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bemgpu  # noqa: E402
from bemgpu import meshes  # noqa: E402

C_WATER = 1500.0
G_WEAK, H_WEAK = 1.0357, 1.0279      # density and sound-speed contrasts of a weak scatterer
EXACT_UNKNOWNS = 11000               # larger dense complex128 solves take too long


# ------------------------------------------------------------------------ the cases
def listed():
    return [
        # one backscatter amplitude read from a solution that is kept: the smallest call
        dict(name="amplitude_1280", kind="far_field", boundary="rigid", precision="double",
             sub=3, a=0.01, ka=1.62, ndir=0),
        # a bistatic pattern of the benchmark's fluid spheroid, many directions at once
        dict(name="pattern_5120", kind="far_field", boundary="fluid", precision="mixed",
             nlon=64, nrings=40, a=0.02, b=0.01, ka=5.5, ndir=6000),
        # the pressure on a cloud of points inside and around a fluid body
        dict(name="field_2880", kind="field", boundary="fluid", precision="mixed",
             nlon=48, nrings=30, a=0.02, b=0.01, ka=4.0, npts=2001),
        # one small solve with the defaults (complex128), as in an interactive session
        dict(name="solve_320_double", kind="solve", boundary="rigid", precision="double",
             sub=2, a=0.01, ka=1.62),
        # the rigid-sphere benchmark, one frequency, one direction
        dict(name="solve_1280_mixed", kind="solve", boundary="rigid", precision="mixed",
             sub=3, a=0.01, ka=1.62),
        # an ordinary fluid body with the default precision (complex128 factor)
        dict(name="fluid_2880_double", kind="solve", boundary="fluid", precision="double",
             nlon=48, nrings=30, a=0.02, b=0.01, ka=4.0),
        # many incidence angles of one large rigid body: one factor, 181 right-hand sides
        dict(name="sweep_20480_mixed", kind="sweep", boundary="rigid", precision="mixed",
             nlon=128, nrings=80, a=0.05, b=0.0125, ka=12.57, nang=181),
        # the benchmark's frequency sweep: 64 frequencies of one fluid body as one batch
        dict(name="freqs_64x5120_mixed", kind="freqs", boundary="fluid", precision="mixed",
             nlon=64, nrings=40, a=0.02, b=0.01, ka_lo=1.0, ka=10.05, count=64),
        # a batch of rigid and soft bodies of very different sizes
        dict(name="bodies_24_mixed", kind="bodies", precision="mixed", count=24, lo=500,
             hi=12000, master=20261204),
        # the compressed operators with GMRES on a large rigid body
        dict(name="hmatrix_20480_mixed", kind="hmatrix", boundary="rigid", precision="mixed",
             nlon=128, nrings=80, a=0.05, b=0.0125, ka=12.57),
        # the Nyström discretisation of the rigid sphere (7 unknowns per panel)
        dict(name="nystrom_1280_mixed", kind="nystrom", boundary="rigid", precision="mixed",
             sub=3, a=0.01, ka=1.62),
        # requests for different bodies handed to the server together
        dict(name="served_10_mixed", kind="served", precision="mixed", count=10, lo=500,
             hi=4000, nfreq=4, nang=16, master=20261205),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _spheroid(rng, lo, hi):
    """Grid, axes and wavenumber of a jittered spheroid of lo..hi panels."""
    aspect = rng.uniform(1.2, 4.0)
    for _ in range(100):
        nlon, nrings = meshes.grid_for_panels(_log_int(rng, lo, hi), aspect)
        if lo <= 2 * nlon * nrings <= hi:
            break
    a = rng.uniform(0.01, 0.05)
    b = a / aspect
    # at least about seven panels per wavelength
    edge = math.sqrt(4.0 * math.pi * a * b / (2 * nlon * nrings) * 2.3)
    ka_hi = min(13.0, 0.85 * a / edge)
    return dict(nlon=nlon, nrings=nrings, a=round(a, 5), b=round(b, 5),
                ka=round(math.exp(rng.uniform(math.log(0.4), math.log(ka_hi))), 4))


def draw(rng):
    kind = rng.choice(["far_field", "field", "solve", "solve", "sweep", "freqs", "bodies",
                       "hmatrix", "nystrom", "served"])
    prec = rng.choice(["double", "mixed"])
    bc = rng.choice(["rigid", "pressure_release", "fluid"])
    two = 2 if bc == "fluid" else 1
    if kind == "far_field":
        return dict(kind=kind, boundary=bc, precision="mixed", ndir=_log_int(rng, 1, 6000),
                    **_spheroid(rng, 320, 5120))
    if kind == "field":
        return dict(kind=kind, boundary=bc, precision="mixed", npts=_log_int(rng, 1, 2001),
                    **_spheroid(rng, 320, 2880))
    if kind == "solve":
        return dict(kind=kind, boundary=bc, precision=prec,
                    **_spheroid(rng, 200, (5760 if prec == "double" else 10240) // two))
    if kind == "sweep":
        bc = rng.choice(["rigid", "pressure_release"])
        return dict(kind=kind, boundary=bc, precision=prec, nang=_log_int(rng, 2, 181),
                    **_spheroid(rng, 500, 3000 if prec == "double" else 20480))
    if kind == "freqs":
        s = _spheroid(rng, 300, 1000 if prec == "double" else 5120)
        return dict(kind=kind, boundary="fluid", precision=prec, ka_lo=round(0.3 * s["ka"], 4),
                    count=_log_int(rng, 2, 8 if prec == "double" else 64), **s)
    if kind == "bodies":
        return dict(kind=kind, precision="mixed", count=rng.randint(2, 24), lo=500,
                    hi=_log_int(rng, 2000, 12000), master=rng.randrange(1 << 30))
    if kind == "hmatrix":
        return dict(kind=kind, boundary="rigid", precision=prec, **_spheroid(rng, 2000, 20480))
    if kind == "nystrom":
        return dict(kind=kind, boundary=bc, precision=prec,
                    **_spheroid(rng, 100, (500 if prec == "double" else 1280) // two))
    return dict(kind=kind, precision="mixed", count=rng.randint(2, 10), lo=500,
                hi=_log_int(rng, 1000, 4000), nfreq=rng.randint(1, 4), nang=_log_int(rng, 1, 16),
                master=rng.randrange(1 << 30))


# ------------------------------------------------------------------------ inputs
def _panels(case):
    return 20 * 4 ** case["sub"] if "sub" in case else 2 * case["nlon"] * case["nrings"]


def _geometry(case, seed):
    if "sub" in case:
        nodes, tris = meshes.icosphere(case["a"], case["sub"])
        u = np.random.default_rng([seed, 7]).uniform(-1.0, 1.0, nodes.shape)
        return nodes + 0.002 * case["a"] * u, tris
    return meshes.uv_spheroid(case["a"], case["b"], case["nlon"], case["nrings"], jitter=0.02,
                              seed=seed + 1)


def _boundary(name):
    if name == "fluid":
        return bemgpu.FluidFilled(G_WEAK, H_WEAK)
    return bemgpu.Rigid() if name == "rigid" else bemgpu.PressureRelease()


def _bodies(case, seed):
    """Bodies of revolution: sizes and aspects belong to the case, shapes, frequencies and
    directions to the seed."""
    rng = np.random.default_rng([seed, 11])
    out = []
    for i in range(case["count"]):
        d = meshes.random_body(case["master"], i, (case["lo"], case["hi"]))
        nodes, tris = meshes.body_of_revolution(d["b"], d["aspect"], rng.uniform(-0.05, 0.05, 4),
                                                d["nlon"], d["nrings"])
        na = 1 + (7 * i) % case.get("nang", 1)
        out.append(dict(nodes=nodes, tris=tris, boundary=d["boundary"],
                        k=2 * math.pi * d["frequency"] / C_WATER * rng.uniform(0.97, 1.03),
                        beta=np.arccos(rng.uniform(-1.0, 1.0, na)),
                        alpha=rng.uniform(0.0, 2 * math.pi, na),
                        nfreq=1 + i % case.get("nfreq", 1)))
    return out


def _inputs(case, seed):
    """Everything that the caller chooses, as host data (the basis of prepare and exact)."""
    if case["kind"] in ("bodies", "served"):
        return dict(bodies=_bodies(case, seed))
    rng = np.random.default_rng([seed, 3])
    nodes, tris = _geometry(case, seed)
    inp = dict(nodes=nodes, tris=tris, k=case["ka"] / case["a"] * rng.uniform(0.98, 1.02),
               beta=float(rng.uniform(0.2, math.pi - 0.2)),
               alpha=float(rng.uniform(0.0, 2 * math.pi)))
    if case["kind"] == "sweep":
        inp["angles"] = np.linspace(0.0, math.pi, case["nang"])
        inp["alpha"] = float(rng.uniform(0.0, 0.5))
    if case["kind"] == "freqs":
        inp["ks"] = np.linspace(case["ka_lo"], case["ka"], case["count"]) / case["a"] * \
            rng.uniform(0.98, 1.02)
    if case["kind"] == "far_field" and case["ndir"]:
        d = rng.normal(size=(case["ndir"], 3))
        inp["dirs"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    if case["kind"] == "field":
        n = case["npts"]
        d = rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        rho = rng.uniform(1.06, 4.0, n)
        if case["boundary"] == "fluid":          # a third of the points inside the body
            rho[::3] = rng.uniform(0.1, 0.9, len(rho[::3]))
        inp["points"] = d * rho[:, None] * np.array([case["a"], case["b"], case["b"]])
        inp["inside"] = rho < 1.0
    return inp


def prepare(case, seed):
    inp = _inputs(case, seed)
    st = dict(case=case, inp=inp)
    if case["kind"] in ("bodies", "served"):
        for b in inp["bodies"]:
            b["surface"] = bemgpu.mesh(b["nodes"], b["tris"])
            b["bc"] = _boundary(b["boundary"])
        if case["kind"] == "served":             # distinct requests: no factor is met twice
            st["server"] = bemgpu.Server(max_batch=64, cache_bytes=1, lanes=2)
        return st
    st["surface"] = bemgpu.mesh(inp["nodes"], inp["tris"])
    st["bc"] = _boundary(case["boundary"])
    if case["kind"] in ("far_field", "field"):   # queries of a solution that is kept
        st["sol"] = bemgpu.bem(st["surface"], st["bc"], inp["k"], precision=case["precision"],
                               incidence_angle=inp["beta"], incidence_azimuth=inp["alpha"])
    return st


# ------------------------------------------------------------------------ one pass
def _all_of(sol):
    p, q = sol.traces()
    return dict(amplitude=sol.far_field(), p=p, q=q)


def run(st):
    case, inp, kind = st["case"], st["inp"], st["case"]["kind"]
    if kind == "far_field":
        return st["sol"].far_field(inp.get("dirs"))
    if kind == "field":
        return bemgpu.pressure(st["sol"], inp["points"], field="total")
    if kind in ("solve", "nystrom", "hmatrix"):
        opts = dict(discretization="nystrom") if kind == "nystrom" else \
            dict(compression=dict(method="hmatrix", tol=1e-5)) if kind == "hmatrix" else {}
        sol = bemgpu.bem(st["surface"], st["bc"], inp["k"], precision=case["precision"],
                         incidence_angle=inp["beta"], incidence_azimuth=inp["alpha"], **opts)
        out = _all_of(sol)
        sol.close()
        return out
    if kind == "sweep":
        r = bemgpu.incidence_angle_sweep(st["surface"], st["bc"], inp["k"], inp["angles"],
                                         incidence_azimuth=inp["alpha"],
                                         precision=case["precision"])
        return dict(amplitudes=r.amplitudes, target_strength=r.target_strength)
    if kind == "served":
        srv = st["server"]
        tickets = []
        for b in inp["bodies"]:
            ks = b["k"] * np.linspace(0.6, 1.0, b["nfreq"]) if b["nfreq"] > 1 else [b["k"]]
            tickets.append(srv.submit(b["surface"], b["bc"], ks, b["beta"], b["alpha"],
                                      precision=case["precision"]))
        return [srv.wait(t)[0] for t in tickets]
    # batches: every system assembled and factored together, then solved together
    opts = dict(precision=case["precision"])
    if kind == "freqs":
        items = [(st["surface"], st["bc"], k, opts) for k in inp["ks"]]
        beta, alpha = [[inp["beta"]]] * len(items), [[inp["alpha"]]] * len(items)
    else:
        items = [(b["surface"], b["bc"], b["k"], opts) for b in inp["bodies"]]
        beta, alpha = [b["beta"] for b in inp["bodies"]], [b["alpha"] for b in inp["bodies"]]
    factors = bemgpu.factor_batch(items)
    sols = bemgpu.solve_batch(factors, beta, alpha)
    if kind == "freqs":
        out = dict(amplitudes=np.concatenate([s.far_field() for s in sols]))
        out["p"], out["q"] = sols[-1].traces()
    else:
        out = [_all_of(s) if i < 16 else s.far_field() for i, s in enumerate(sols)]
    for x in sols + factors:
        x.close()
    return out


# ------------------------------------------------------------------------ work of one pass
_PAIR = 7 * 60.0      # flops of the four kernels of one panel pair at its seven points


def _solve_work(boundary, n, nrhs=1, nodes=1):
    """Dense path: operators of every pair, LU, one forward and back substitution each."""
    N = n * nodes
    kinds, m = (2, 2 * N) if boundary == "fluid" else (1, N)
    pair = _PAIR if nodes == 1 else _PAIR / 7
    flops = kinds * pair * N * N + 8.0 / 3.0 * m ** 3 + 8.0 * nrhs * float(m) ** 2
    return 8.0 * 3 * 1.5 * n + 16.0 * nrhs * 2 * N, flops


def work(case):
    kind = case["kind"]
    if kind in ("bodies", "served"):
        by = fl = 0.0
        for i in range(case["count"]):
            d = meshes.random_body(case["master"], i, (case["lo"], case["hi"]))
            nf, na = 1 + i % case.get("nfreq", 1), 1 + (7 * i) % case.get("nang", 1)
            b, f = _solve_work("rigid", d["panels"], na)
            by, fl = by + b * nf, fl + f * nf
        return dict(bytes=by, flops=fl)
    n = _panels(case)
    if kind == "far_field":
        nd = max(1, case["ndir"])
        return dict(bytes=n * (7 * 24 + 24 + 32.0) + nd * 40.0, flops=n * nd * 7 * 40.0)
    if kind == "field":
        return dict(bytes=n * (7 * 24 + 24 + 32.0) + case["npts"] * 40.0,
                    flops=n * case["npts"] * 7 * 50.0)
    if kind == "hmatrix":     # about 2200 stored entries a row, 100 products, one basis each
        return dict(bytes=100.0 * 2200 * n * 8, flops=100.0 * (8.0 * 2200 * n + 16.0 * 50 * n))
    if kind == "sweep":
        b, f = _solve_work(case["boundary"], n, case["nang"])
    elif kind == "freqs":
        b, f = _solve_work(case["boundary"], n)
        b, f = b * case["count"], f * case["count"]
    else:
        b, f = _solve_work(case["boundary"], n, 1, 7 if kind == "nystrom" else 1)
    return dict(bytes=b, flops=f)


# ------------------------------------------------------------------------ 64-bit values
# Radon's seven-point rule of degree five: barycentric coordinates and weights
_S15 = math.sqrt(15.0)
_RA, _RB_ = (6 - _S15) / 21, (6 + _S15) / 21
_RULE = [(1 / 3, 1 / 3, 1 / 3)] + \
    [(1 - 2 * _RB_, _RB_, _RB_), (_RB_, 1 - 2 * _RB_, _RB_), (_RB_, _RB_, 1 - 2 * _RB_)] + \
    [(1 - 2 * _RA, _RA, _RA), (_RA, 1 - 2 * _RA, _RA), (_RA, _RA, 1 - 2 * _RA)]
_WRULE = [0.225] + [(155 + _S15) / 1200] * 3 + [(155 - _S15) / 1200] * 3
_FOURPI = 4.0 * math.pi


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Surface:
    """Panel geometry: vertices, centroids, unit normals, areas, diameters, Gauss points."""

    def __init__(self, nodes, tris):
        t = torch.as_tensor(np.asarray(tris).T - 1, device=_dev())
        self.v = torch.as_tensor(np.ascontiguousarray(np.asarray(nodes).T), device=_dev())[t]
        cr = torch.linalg.cross(self.v[:, 1] - self.v[:, 0], self.v[:, 2] - self.v[:, 0])
        ln = cr.norm(dim=1)
        self.n, self.area, self.c = cr / ln[:, None], 0.5 * ln, self.v.mean(dim=1)
        self.diam = (self.v.roll(-1, 1) - self.v).norm(dim=2).max(dim=1).values
        self.bary = torch.tensor(_RULE, dtype=torch.float64, device=_dev())
        self.g = torch.einsum("qa,pad->pqd", self.bary, self.v)
        self.w = torch.tensor(_WRULE, dtype=torch.float64, device=_dev())


def _kernels(k, u, nx, ny, w):
    """Weighted S, D, K', H at u = y - x (regular points)."""
    r = (u * u).sum(-1).sqrt()
    z = k * r
    e = torch.complex(z.cos(), z.sin()) * (w / (_FOURPI * r))
    iz = 1j * z
    uy, ux, nn = (u * ny).sum(-1) / r, (u * nx).sum(-1) / r, (nx * ny).sum(-1)
    gp = e * (iz - 1.0) / r
    return e, gp * uy, -gp * ux, e / (r * r) * ((1 - iz) * nn - (3 - 3 * iz - z * z) * ux * uy)


def _remainder(k, u, nx, ny, w):
    """Helmholtz minus Laplace kernels (H also minus (k^2/2)(nx.ny) G0)."""
    r = (u * u).sum(-1).sqrt()
    z = k * r
    e = torch.complex(z.cos(), z.sin())
    iz = 1j * z
    e0, e1 = e - 1.0, e * (1 - iz) - 1.0 - 0.5 * z * z
    e2, e3 = e * (iz - 1) + 1.0, e * (3 - 3 * iz - z * z) - 3.0
    t = torch.ones_like(iz)
    s0, s1, s2, s3 = (torch.zeros_like(iz) for _ in range(4))
    for m in range(1, 25):                       # the series where the closed forms cancel
        t = t * iz / m
        s0, s2, s3 = s0 + t, s2 + (m - 1) * t, s3 + (m - 1) * (m - 3) * t
        if m >= 3:
            s1 = s1 + (1 - m) * t
    small = z < 0.5
    e0, e1, e2, e3 = (torch.where(small, s, x) for s, x in
                      ((s0, e0), (s1, e1), (s2, e2), (s3, e3)))
    uy, ux, nn = (u * ny).sum(-1) / r, (u * nx).sum(-1) / r, (nx * ny).sum(-1)
    a = w / (_FOURPI * r)
    return a * e0, a / r * e2 * uy, -a / r * e2 * ux, a / (r * r) * (e1 * nn - e3 * ux * uy)


def _laplace(v, n, x, nx, self_panel):
    """Closed forms of the Laplace S, D, K', H of flat triangles v at the points x."""
    pint, hs, gp = 0.0, 0.0, 0.0
    for a in range(3):
        pa, pb = v[:, a], v[:, (a + 1) % 3]
        e = pb - pa
        ln = e.norm(dim=1)
        s = e / ln[:, None]
        m = torch.linalg.cross(s, n)
        w, wb = x - pa, x - pb
        sm = -(w * s).sum(1)
        sp = ln + sm
        t0, dpl = -(w * m).sum(1), (w * n).sum(1)
        rm, rp = w.norm(dim=1), wb.norm(dim=1)
        f = torch.where(sm >= 0, ((rp + sp) / (rm + sm)).log(),
                        torch.where(sp <= 0, ((rm - sm) / (rp - sp)).log(),
                                    ((rp + sp) * (rm - sm) / (t0 * t0 + dpl * dpl)).log()))
        pint, gp = pint + t0 * f, gp - m * f[:, None]
        sw = torch.linalg.cross(s, w)
        rho2 = (sw * sw).sum(1)
        on_line = rho2 <= 1e-24 * ln * ln
        hs = hs + torch.where(on_line, 0.0, (nx * sw).sum(1) / torch.where(on_line, 1.0, rho2) *
                              (sp / rp - sm / rm))
    r = v - x[:, None, :]
    rn = r.norm(dim=2)
    num = (r[:, 0] * torch.linalg.cross(r[:, 1], r[:, 2])).sum(1)
    den = rn.prod(dim=1) + (r[:, 0] * r[:, 1]).sum(1) * rn[:, 2] + \
        (r[:, 0] * r[:, 2]).sum(1) * rn[:, 1] + (r[:, 1] * r[:, 2]).sum(1) * rn[:, 0]
    om = torch.where(self_panel, 0.0, 2.0 * torch.atan2(num, den))
    d = torch.where(self_panel, 0.0, ((x - v[:, 0]) * n).sum(1))
    return ((pint + d * om) / _FOURPI, -om / _FOURPI,
            ((nx * gp).sum(1) + (nx * n).sum(1) * om) / _FOURPI, -hs / _FOURPI)


def _operators(P, k, x=None, nx=None, rows=512):
    """S, D, K', H of every panel at the points x (default: the centroids)."""
    own = x is None
    x, nx = (P.c, P.n) if own else (x, nx)
    out = [torch.empty(len(x), len(P.c), dtype=torch.complex128, device=x.device)
           for _ in range(4)]
    for r0 in range(0, len(x), rows):
        xs, ns = x[r0:r0 + rows], nx[r0:r0 + rows]
        acc = [0.0] * 4
        for q in range(7):
            u = P.g[None, :, q, :] - xs[:, None, :]
            t = _kernels(k, u, ns[:, None, :], P.n[None, :, :], P.w[q] * P.area[None, :])
            acc = [p + o for p, o in zip(acc, t)]
        d = xs[:, None, :] - P.c[None, :, :]
        near = (d * d).sum(-1) < 4.0 * (P.diam * P.diam)[None, :]
        if own:
            near[torch.arange(len(xs)), torch.arange(r0, r0 + len(xs))] = True
        i, j = near.nonzero(as_tuple=True)
        slf = (i + r0 == j) if own else torch.zeros_like(i, dtype=torch.bool)
        xi, ni, nj, vj = xs[i], ns[i], P.n[j], P.v[j]
        val = list(_laplace(vj, nj, xi, ni, slf))
        val[3] = val[3] + 0.5 * k * k * (ni * nj).sum(1) * val[0]
        val = [t.to(torch.complex128) for t in val]
        o = (~slf).nonzero()[:, 0]
        for q in range(7):
            t = _remainder(k, P.g[j[o], q] - xi[o], ni[o], nj[o], P.w[q] * P.area[j[o]])
            for p, y in zip(val, t):
                p[o] += y
        s = slf.nonzero()[:, 0]                  # the own panel, split at its centroid
        for a in range(3):
            for q in range(7):
                b = _RULE[q]
                y = b[0] * P.c[j[s]] + b[1] * vj[s, a] + b[2] * vj[s, (a + 1) % 3]
                t = _remainder(k, y - xi[s], ni[s], nj[s], P.w[q] * P.area[j[s]] / 3.0)
                for p, z in zip(val, t):
                    p[s] += z
        for p, z, dst in zip(acc, val, out):
            p[i, j] = z
            dst[r0:r0 + len(xs)] = p
    return out


_WAVES = torch.tensor([(3, 1, -1), (-3, -2, 2), (-3, 1, -1), (1, 2, -3), (2, 2, 3), (0, 1, 2),
                       (0, -1, -1), (-1, -3, 1), (-3, -3, -1)], dtype=torch.float64)


def _node_operators(P, k, rows=1024):
    """S, D, K', H on the quadrature nodes with the plane-wave correction of each element."""
    y, ny = P.g.reshape(-1, 3), P.n.repeat_interleave(7, 0)
    w = (P.area[:, None] * P.w[None, :]).reshape(-1)
    N, out = len(w), []
    out = [torch.empty(N, N, dtype=torch.complex128, device=y.device) for _ in range(4)]
    for r0 in range(0, N, rows):
        u = y[None, :, :] - y[r0:r0 + rows, None, :]
        i = torch.arange(len(u), device=y.device)
        u[i, i + r0] = 1.0
        t = _kernels(k, u, ny[r0:r0 + rows, None, :], ny[None, :, :], w[None, :])
        for dst, o in zip(out, t):
            o[i, i + r0] = 0.0
            dst[r0:r0 + len(u)] = o
    S, D, K, H = out
    dirs = (_WAVES / _WAVES.norm(dim=1, keepdim=True)).to(y.device)
    u = (1j * k * (y @ dirs.T)).exp()
    f = 1j * k * (ny @ dirs.T) * u
    M = torch.cat([u.reshape(-1, 7, 9), f.reshape(-1, 7, 9)], dim=1)
    sc = M.abs().square().sum(2).sqrt()
    pinv = torch.linalg.pinv((M / sc[:, :, None]).transpose(1, 2), rtol=1e-13)
    e = torch.arange(N // 7, device=y.device) * 7
    blk = e[:, None] + torch.arange(7, device=y.device)[None, :]
    for mult, A, B in ((u, S, D), (f, K, H)):
        defect = (-0.5 * mult + A @ f - B @ u).reshape(-1, 7, 9)
        W = torch.einsum("eiq,etq->eti", pinv, defect) / sc[:, None, :]
        B[blk[:, :, None], blk[:, None, :]] += W[:, :, :7]
        A[blk[:, :, None], blk[:, None, :]] -= W[:, :, 7:]
    return S, D, K, H


def _far(P, k, dirs, p, q, nodes=False):
    out = []
    for d in dirs.split(64):
        ph = (-1j * k * torch.einsum("pqd,md->mpq", P.g, d)).exp() * P.w * P.area[:, None]
        dn = 1j * k * (d @ P.n.T)
        if nodes:
            s = dn[:, :, None] * p.reshape(1, -1, 7) + q.reshape(1, -1, 7)
            out.append(-(ph * s).sum((1, 2)) / _FOURPI)
        else:
            out.append(-(ph.sum(2) * (dn * p + q)).sum(1) / _FOURPI)
    return torch.cat(out)


def _direction(beta, alpha):
    return torch.tensor([math.cos(beta), math.sin(beta) * math.cos(alpha),
                         math.sin(beta) * math.sin(alpha)], dtype=torch.float64, device=_dev())


def _traces(P, boundary, k, angles, nodes=False):
    """Scattered traces (one column per direction) and the backscatter amplitudes."""
    y, ny = (P.g.reshape(-1, 3), P.n.repeat_interleave(7, 0)) if nodes else (P.c, P.n)
    ops = _node_operators if nodes else _operators
    d = torch.stack([_direction(b, a) for b, a in angles])
    pin = (1j * k * (y @ d.T)).exp()
    qin = 1j * k * (ny @ d.T) * pin
    S, D, K, H = ops(P, k)
    eye = torch.eye(len(y), dtype=torch.complex128, device=y.device)
    al = 1j / k
    if boundary == "fluid":
        Si, Di, Ki, Hi = ops(P, k / H_WEAK)
        A = torch.cat([torch.cat([eye - D + Di, S - G_WEAK * Si], 1),
                       torch.cat([-H + Hi / G_WEAK, eye + K - Ki], 1)], 0)
        x = torch.linalg.solve(A, torch.cat([pin, qin]))
        p, q = x[:len(y)] - pin, x[len(y):] - qin
    else:
        M1, M2 = 0.5 * eye - D - al * H, S + al * (0.5 * eye + K)
        if boundary == "rigid":
            p, q = torch.linalg.solve(M1, M2 @ qin), -qin
        else:
            p, q = -pin, torch.linalg.solve(M2, M1 @ pin)
    amp = torch.cat([_far(P, k, -d[i:i + 1], p[:, i], q[:, i], nodes) for i in range(len(d))])
    return p, q, amp, pin, qin


def exact(case, seed):
    kind, inp = case["kind"], _inputs(case, seed)
    if kind in ("bodies", "served"):             # one of the smaller bodies stands for all
        out = [None] * case["count"]
        sizes = [b["tris"].shape[1] for b in inp["bodies"]]
        for i in (int(np.argmin(sizes)), int(np.argsort(sizes)[len(sizes) // 2])):
            b = inp["bodies"][i]
            if sizes[i] > 6000 or (kind == "served" and b["nfreq"] > 2):
                continue
            ks = b["k"] * np.linspace(0.6, 1.0, b["nfreq"]) if b["nfreq"] > 1 else [b["k"]]
            P = _Surface(b["nodes"], b["tris"])
            r = [_traces(P, b["boundary"], float(k), list(zip(b["beta"], b["alpha"])))
                 for k in ks]
            if kind == "served":
                out[i] = torch.stack([x[2] for x in r])
            elif i < 16:
                out[i] = dict(amplitude=r[0][2], p=r[0][0][:, 0], q=r[0][1][:, 0])
            else:
                out[i] = r[0][2]
        return out if any(x is not None for x in out) else None
    nodes = kind == "nystrom"
    m = _panels(case) * (7 if nodes else 1) * (2 if case["boundary"] == "fluid" else 1)
    if m > EXACT_UNKNOWNS:
        return None
    P, k = _Surface(inp["nodes"], inp["tris"]), inp["k"]
    if kind == "sweep":
        amp = _traces(P, case["boundary"], k, [(b, inp["alpha"]) for b in inp["angles"]])[2]
        return dict(amplitudes=amp, target_strength=20 * amp.abs().log10())
    if kind == "freqs":                          # the traces of the highest frequency
        p, q = _traces(P, case["boundary"], float(inp["ks"][-1]),
                       [(inp["beta"], inp["alpha"])])[:2]
        return dict(amplitudes=None, p=p[:, 0], q=q[:, 0])
    p, q, amp, pin, qin = _traces(P, case["boundary"], k, [(inp["beta"], inp["alpha"])], nodes)
    if kind == "far_field":
        if "dirs" not in inp:
            return amp
        return _far(P, k, torch.as_tensor(inp["dirs"], device=_dev()), p[:, 0], q[:, 0])
    if kind == "field":
        x = torch.as_tensor(inp["points"], device=_dev())
        ins = torch.as_tensor(inp["inside"], device=_dev())
        val = torch.empty(len(x), dtype=torch.complex128, device=_dev())
        S, D, _, _ = _operators(P, k, x[~ins], torch.zeros_like(x[~ins]))
        val[~ins] = (D @ p - S @ q)[:, 0] + \
            (1j * k * (x[~ins] @ _direction(inp["beta"], inp["alpha"]))).exp()
        if bool(ins.any()):
            S, D, _, _ = _operators(P, k / H_WEAK, x[ins], torch.zeros_like(x[ins]))
            val[ins] = (S @ (G_WEAK * (q + qin)) - D @ (p + pin))[:, 0]
        return val
    return dict(amplitude=amp, p=p[:, 0], q=q[:, 0])
