"""The exact mode's quotients by shared divisors (five fused multiply-adds from a correctly rounded
reciprocal, or an IEEE division where exponents are extreme) and its Barth ratio (one division of
the smallest fraction): gradients, fluxes and residuals bit for bit equal to the CPU oracle, on
states whose differences are ordinary, zero, all but equal, or outside the range of either form.
"""
import numpy as np
import pytest

import oracle_py as op

pytestmark = pytest.mark.gpu


def states(kind, nc, rng):
    q = np.empty((5, nc))
    q[0], q[1] = 1.0 + 0.3 * rng.random(nc), 1.0 + 0.3 * rng.random(nc)
    q[2:] = 0.4 * rng.standard_normal((3, nc))
    if kind == "zero":           # uniform pressure, one velocity component 0, another constant
        q[1], q[3], q[4] = 1.0, 0.0, 0.25
    elif kind == "equal":        # differences of a few units in the last place: ties of the ratio
        q = np.array([1.0, 1.0, 0.5, -0.5, 0.25])[:, None] * (1.0 + 2.2e-16 * rng.integers(0, 3, (5, nc)))
    elif kind == "tiny":         # velocity differences below 2^-700, one component subnormal
        q[2] *= 1e-230
        q[3] *= 1e-310
        q[4, ::2] *= 1e-215
    elif kind == "scaled":       # densities and pressures around 1e-90
        q[:2] *= 1e-90
    elif kind == "wide":         # speeds 1e-70 to 1, both sides of FP32's range
        q[2:] *= 10.0 ** rng.uniform(-70, 0, (3, nc))
    elif kind == "supersonic":   # waves inside and outside the entropy fix
        q[2:] = 2.0 * rng.standard_normal((3, 1)) + 0.2 * rng.standard_normal((3, nc))
    return q


@pytest.mark.parametrize("kind", ["ordinary", "zero", "equal", "tiny", "scaled", "wide", "supersonic"])
@pytest.mark.parametrize("scheme,highres,limiter,postlim", [("ROE", "MUSCL-UNS", "NONE", "BARTH"),
                                                            ("ROE", "MUSCL", "NONE", "SUPERBARTH"),
                                                            ("ROE", "MUSCL", "ALBADA", "NONE"),
                                                            ("HLLC", "MUSCL-FAST", "MINMOD", "NONE")])
def test_bitwise(kind, scheme, highres, limiter, postlim):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from typhon_gb300 import build
    build.build()
    import typhon_gb300 as ty
    raw = ty.gen_tet_box(4, 1.0, jitter=0.1, seed=3)
    bcs = ty.periodic_box_bcs((1.0,) * 3)
    md = ty.preprocess(raw, 3, bcs)
    om = op.Mesh.from_raw(raw).build(3, bcs)
    prim = states(kind, md.ncell, np.random.default_rng(8))
    g = ty.Grid(md)
    g.set_spat(scheme, highres, limiter, postlim, gradmeth="LSQ", mode="exact")
    g.set_prim(prim)
    s = op.Solver(om, {"ROE": op.SCH_ROE, "HLLC": op.SCH_HLLC}[scheme],
                  {"MUSCL": op.HRES_MUSCL, "MUSCL-UNS": op.HRES_MUSCLUNS, "MUSCL-FAST": op.HRES_MUSCLFAST}[highres],
                  {"NONE": op.LIM_NONE, "ALBADA": op.LIM_ALBADA, "MINMOD": op.LIM_MINMOD}[limiter],
                  {"NONE": op.POSTLIM_NONE, "BARTH": op.POSTLIM_BARTH, "SUPERBARTH": op.POSTLIM_SUPERBARTH}[postlim],
                  op.GRAD_LSQ, rk="RK2", cfl=0.8)
    s.set_prim(prim)
    R = g.integration_grid(1e-3)
    s.rhs(1e-3)
    n = md.ncell_int
    assert np.isfinite(R).all()
    assert np.array_equal(g.debug("grad")[:, :n], s.get("grad")[:, :n])
    assert np.array_equal(g.debug("flux"), s.get("flux"))
    assert np.array_equal(R, s.get("residu")[:, :n])
    g.close()
