"""Conjugate gradients of heat conduction at the edges: data so small that r.D^-1 r is subnormal,
few cells, where the residual becomes exactly zero between two checks of it, and the continuation and
the mixed form's change of matrix in every storage form of the vectors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ty():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from typhon_gb300 import build
    build.build()
    import typhon_gb300
    return typhon_gb300


def setup(ty, n, sigma):
    """n^3 x 6 tetrahedra, lognormal conductivity, zero temperature on the x faces, adiabatic elsewhere."""
    from typhon_gb300 import umesh
    md = ty.preprocess(umesh.gen_kuhn_box(n, 1.0), 3, [(f, umesh.BC_WALL, "", (0.0, 0.0, 0.0)) for f in
                                                       ("IMIN", "IMAX", "JMIN", "JMAX", "KMIN", "KMAX")])
    kind = np.zeros(md.nface, np.int32)
    b = np.arange(md.nface_int, md.nface)
    kind[b] = np.where(np.abs(md.face_centre[b, 0] - 0.5) > 0.4999, 1, 2)
    g = ty.Grid(md)
    g.set_spat("HLLC", mode="fast")
    kc = np.exp(sigma * np.random.default_rng(n).standard_normal(md.ncell_int))
    g.kdif_setup(kc, kind, np.zeros(md.nface), flux="FULL", heat_capacity=1.0)
    return md, g


def residual(md, g, x, b):
    """|b - S x| / |b| on the assembled symmetrised matrix."""
    a, c1, c2 = g.kdif_get("jac")[:md.nface_int], md.fc1[:md.nface_int], md.fc2[:md.nface_int]
    n = len(x)
    y = g.kdif_get("diag") * x + np.bincount(c1, a * x[c2], n) + np.bincount(c2, a * x[c1], n)
    return np.linalg.norm(b - y) / np.linalg.norm(b)


# |b|^2 is about 1e-303; where |r| / |b| has fallen to 1e-5, gamma = r.D^-1 r is below 2^-1022 and still
# has 2^-1074 / 1e-313 = 5e-11 relative precision.  Tolerance: the requested 1e-5, and as much again
# for the recurrence's drift from the true residual.
@pytest.mark.parametrize("solver", ["CG"])
def test_subnormal_gamma(ty, solver):
    md, g = setup(ty, 8, 2.0)
    scale = 1e-153
    g.kdif_set_temperature(scale * np.random.default_rng(1).uniform(0.0, 1.0, md.ncell_int))
    T0 = g.kdif_temperature()
    st = g.kdif_implicit_step(0.05, solver, tol=1e-5, max_it=2000)
    assert st["iterations"] < 2000 and st["rel_res"] < 1e-5
    x = (g.kdif_temperature() - T0) / scale
    assert np.isfinite(x).all() and np.abs(x).max() > 0
    assert residual(md, g, x, g.kdif_get("balance") / scale) < 2e-5
    g.close()


# One cell: one step solves the system and leaves r = 0 or rounding.  A strip of equal cells, heated
# alike along both sides: equal rows, the same.  Checked every ten iterations, the solve must end at
# the next check and not carry 0 / 0 into x.  Tolerance: 1e-12 is requested; the true residual of a
# well-conditioned system of a few cells is within a few ulp of the recurrence's.
@pytest.mark.parametrize("solver", ["CG", "CG-MIXED"])
@pytest.mark.parametrize("cells", ["one", "strip"])
@pytest.mark.parametrize("seed", range(8))
def test_exact_convergence(ty, cells, solver, seed):
    from typhon_gb300 import umesh
    rng = np.random.default_rng(seed)
    ni = 1 if cells == "one" else 6
    md = ty.preprocess(umesh.gen_grid2d(ni, 1, 1.0, rng.uniform(0.5, 2.0), "quad"), 2,
                       [(f, umesh.BC_WALL, "", (0.0, 0.0, 0.0)) for f in ("IMIN", "IMAX", "JMIN", "JMAX")])
    kind, val = np.zeros(md.nface, np.int32), np.zeros(md.nface)
    b = np.arange(md.nface_int, md.nface)
    y = np.abs(md.face_normal[b, 1]) > 0.5  # the long sides: isothermal; the ends: adiabatic
    kind[b], val[b] = np.where(y, 1, 2), np.where(y, rng.uniform(0.5, 2.0), 0.0)
    g = ty.Grid(md)
    g.set_spat("HLLC", mode="fast")
    g.kdif_setup(np.full(ni, rng.uniform(0.1, 10.0)), kind, val, flux="COMPACT", heat_capacity=rng.uniform(0.5, 2.0))
    cp = g._kdif_cp
    g.kdif_set_temperature(np.full(ni, rng.uniform(0.0, 1.0)))
    T0 = g.kdif_temperature()
    st = g.kdif_implicit_step(rng.uniform(0.1, 1.0), solver, tol=1e-12, max_it=2000)
    T = g.kdif_temperature()
    assert np.isfinite(T).all() and np.isfinite(st["rel_res"]) and st["rel_res"] < 1e-12 and st["iterations"] <= 30
    assert residual(md, g, (T - T0) * cp, g.kdif_get("balance")) < 1e-10
    g.close()


# Two and six cells per thread in registers, and vectors in memory (n = 56): more iterations than a
# launch runs, and the mixed form's restart on the FP64 conductances from the true residual.  Tolerance: the recurrence's
# residual drifts from the true one by rounding times the iterations (1e-16 x 1e4 x a growth of 1e4).
@pytest.mark.parametrize("solver", ["CG", "CG-MIXED"])
@pytest.mark.parametrize("n", [24, 42, 56])
def test_continuation(ty, n, solver):
    md, g = setup(ty, n, 3.0)
    T0 = np.random.default_rng(n).uniform(0.0, 1.0, md.ncell_int)
    g.kdif_set_temperature(T0)
    st = g.kdif_implicit_step(1e3, solver, tol=1e-9, max_it=20000)
    assert st["iterations"] > 1000 and st["rel_res"] < 1e-9
    assert st["refinements"] == (1 if solver == "CG-MIXED" else 0)
    assert residual(md, g, g.kdif_temperature() - T0, g.kdif_get("balance")) < 1e-7
    g.close()
