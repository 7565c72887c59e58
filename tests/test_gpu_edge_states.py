"""States at the edges of the number range, in the fast mode against the CPU oracle or the exact mode.

Tolerance: the fast mode's envelope against the oracle, 1e-12 relative L2 per conserved variable,
unless a test derives its own.
"""
import numpy as np
import pytest

import oracle_py as op

pytestmark = pytest.mark.gpu

RTOL = 1e-12


@pytest.fixture(scope="module")
def ty():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from typhon_gb300 import build
    build.build()
    import typhon_gb300
    return typhon_gb300


def tet_box(ty, n=4):
    raw, bcs = ty.gen_tet_box(n, 1.0, jitter=0.05, seed=3), ty.periodic_box_bcs((1.0,) * 3)
    return raw, bcs, ty.preprocess(raw, 3, bcs)


def close(a, b):
    for rows in ([0], [1], [2, 3, 4]):
        err = np.linalg.norm(a[rows] - b[rows]) / np.linalg.norm(b[rows])
        assert err < RTOL, (rows, err)


# A transverse velocity of subnormal or nearly subnormal size, as in the numerical tail ahead of a
# disturbance.  Subnormal increments carry 2^-1074 / 2e-309 = 2.5e-15 relative rounding each, and the
# common ratio of the velocities passes it on to the increments of u (a few percent of u): about 1e-15.
@pytest.mark.parametrize("size", [2e-309, 1e-307, 1e-200])
@pytest.mark.parametrize("highres,limiter,postlim", [("MUSCL-UNS", "NONE", "BARTH"), ("MUSCL", "NONE", "SUPERBARTH"),
                                                     ("MUSCL", "VAN_LEER", "BARTH")])
def test_barth_subnormal_velocity(ty, highres, limiter, postlim, size):
    raw, bcs, md = tet_box(ty)
    rng = np.random.default_rng(2)
    x = md.cell_centre
    q = np.stack([1.0 + 0.1 * np.sin(2 * np.pi * x[:, 0]), 2.0 + 0.2 * np.cos(2 * np.pi * x[:, 1]),
                  0.5 + 0.1 * np.sin(2 * np.pi * x[:, 1]), size * rng.standard_normal(len(x)), np.zeros(len(x))])
    q[:3] *= 1.0 + 0.02 * rng.standard_normal((3, len(x)))
    g = ty.Grid(md)
    g.set_spat("ROE", highres, limiter, postlim, mode="fast")
    om = op.Mesh.from_raw(raw).build(3, [tuple(b) for b in bcs])
    s = op.Solver(om, op.SCH_ROE, {"MUSCL": op.HRES_MUSCL, "MUSCL-UNS": op.HRES_MUSCLUNS}[highres],
                  {"NONE": op.LIM_NONE, "VAN_LEER": op.LIM_VLEER}[limiter],
                  {"BARTH": op.POSTLIM_BARTH, "SUPERBARTH": op.POSTLIM_SUPERBARTH}[postlim], op.GRAD_LSQ, rk="RK2", cfl=0.5)
    s.set_prim(q)
    dt = s.timestep()
    g.set_prim(q)
    R = g.integration_grid(dt)
    s.rhs(dt)
    close(R, s.get("residu")[:, :md.ncell_int])
    g.close()


# Cells of zero pressure (an evacuated region): T = 0 at the faces between them, where Sutherland's
# viscosity is 0.  The inviscid flux is Rusanov's, regular there.
@pytest.mark.parametrize("flux", ["CELL-AVERAGE", "FULL"])
def test_sutherland_zero_temperature(ty, flux):
    raw, bcs, md = tet_box(ty)
    rng = np.random.default_rng(4)
    x = md.cell_centre
    q = np.stack([1.2 + 0.1 * rng.random(len(x)), 1e5 * (1.0 + 0.1 * rng.random(len(x))), 30.0 * rng.standard_normal(len(x)),
                  20.0 * rng.standard_normal(len(x)), 10.0 * rng.standard_normal(len(x))])
    q[1:, np.linalg.norm(x - 0.5, axis=1) < 0.35] = 0.0  # at rest: p = 0 exactly from the conserved state
    visc = dict(rgas=287.0, prandtl=0.72)
    g = ty.Grid(md)
    g.set_spat("RUSANOV", mode="fast", dissipative_flux=flux, viscosity="SUTHERLAND", **visc)
    om = op.Mesh.from_raw(raw).build(3, [tuple(b) for b in bcs])
    s = op.Solver(om, op.SCH_RUSANOV, gradmeth=op.GRAD_LSQ, viscous={"CELL-AVERAGE": op.VISC_CELLAVG, "FULL": op.VISC_CELLFULL}[flux],
                  visc_law=1, **visc)
    s.set_prim(q)
    g.set_prim(q)
    s.rhs(1e-6)
    b = s.get("residu")[:, :md.ncell_int]
    assert np.isfinite(b).all()
    close(g.integration_grid(1e-6), b)
    g.close()


# Cells of negative pressure, single and side by side: Rusanov's wave speed is the ordinary neighbour's
# beside a single one and NaN between two, in both modes.  Finite entries: the fast mode's envelope.
def test_rusanov_negative_pressure(ty):
    raw, bcs, md = tet_box(ty)
    rng = np.random.default_rng(6)
    nci = md.ncell_int
    q = np.stack([1.0 + 0.1 * rng.random(nci), 2.0 + 0.2 * rng.random(nci), *(2.5 * rng.standard_normal((3, nci)))])
    q[1, rng.random(nci) < 0.08] *= -1.0
    R = {}
    for mode in ("exact", "fast"):
        g = ty.Grid(md)
        g.set_spat("RUSANOV", mode=mode)
        g.set_prim(q)
        R[mode] = g.integration_grid(1e-3)
        g.close()
    e, f = R["exact"], R["fast"]
    nan = ~np.isfinite(e)
    assert nan.any() and not nan.all()
    assert np.array_equal(nan, ~np.isfinite(f))
    close(np.where(nan, 0.0, f), np.where(nan, 0.0, e))


# The slot tables follow the limiter: LIM03's hold other factors than the homogeneous limiters', so a
# handle that changes between them must give what a new handle gives.
@pytest.mark.parametrize("highres", ["MUSCL", "MUSCL-FAST", "MUSCL-UNS"])
def test_limiter_changes_on_one_handle(ty, highres):
    raw, bcs, md = tet_box(ty)
    rng = np.random.default_rng(8)
    x = md.cell_centre
    q = np.stack([1.0 + 0.1 * np.sin(2 * np.pi * x[:, 0]), 2.0 + 0.2 * np.cos(2 * np.pi * x[:, 1]), 0.3 * np.sin(2 * np.pi * x[:, 1]),
                  0.1 * np.cos(2 * np.pi * x[:, 0]), 0.2 * np.sin(2 * np.pi * x[:, 2])])
    q = (q * (1.0 + 0.02 * rng.standard_normal(q.shape)))[:, :md.ncell_int]
    g = ty.Grid(md)
    for limiter in ("ALBADA", "LIM03", "VAN_LEER", "LIM03"):
        R = []
        for h in (g, ty.Grid(md)):
            h.set_spat("HLLC", highres, limiter, mode="fast")
            h.set_prim(q)
            R.append(h.integration_grid(1e-3))
        assert np.array_equal(*R), limiter
    g.close()


# Cells of zero pressure at rest in an adjoint: the derivative of their sound speed is infinite, so their
# own entries have no value in either mode; their neighbours' do.  Finite entries: 1e-11 relative L2 (the
# fast reverse forms against the exact ones on smooth data: a few 1e-15, amplified where al is small).
def test_adjoint_zero_pressure(ty):
    import torch
    from typhon_gb300 import _capi
    raw, bcs, md = tet_box(ty)
    nci = md.ncell_int
    rng = np.random.default_rng(9)
    q = np.stack([1.0 + 0.1 * rng.random(nci), 2.0 + 0.2 * rng.random(nci), *(0.5 * rng.standard_normal((3, nci)))])
    q[1:, rng.random(nci) < 0.05] = 0.0
    lam = torch.as_tensor(rng.standard_normal((5, nci)), device="cuda")
    v = {}
    for mode in ("exact", "fast"):
        g = ty.Grid(md)
        g.set_spat("HLLC", mode=mode)
        g.set_prim(q)
        out = torch.empty_like(lam)
        torch.cuda.synchronize()
        _capi.check(g.lib.ty_adjoint_vjp(g.h, 1e-3, lam.data_ptr(), out.data_ptr()), "ty_adjoint_vjp")
        g.synchronize()
        v[mode] = out.cpu().numpy()
        g.close()
    e, f = v["exact"], v["fast"]
    nan = ~np.isfinite(e)
    assert nan.any() and not nan.all()
    assert np.array_equal(nan, ~np.isfinite(f))
    e, f = np.where(nan, 0.0, e), np.where(nan, 0.0, f)
    assert np.linalg.norm(f - e) < 1e-11 * np.linalg.norm(e)
