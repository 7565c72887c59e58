"""The fast mode's face fluxes against the exact mode's on random states from Mach 0 to 3, which
take every branch: Roe's summed acoustic waves and the call for supersonic faces and those
inside the entropy fix, HLLC's four wave patterns and its wave-speed variants, Rusanov's two
sides, and the viscous flux with both face gradients and both viscosity laws.

Tolerance per variable: 1e-12 of the largest flux (about a hundred FP64 operations whose terms
are at most a few times the flux; an ulp is 1.1e-16).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grids():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from typhon_gb300 import build
    build.build()
    import typhon_gb300 as ty
    out = {}
    for name, raw, dim, bcs in (("tet", ty.gen_tet_box(4, 1.0, jitter=0.05, seed=2), 3, ty.periodic_box_bcs((1.0,) * 3)),
                                ("plate", ty.umesh.gen_flatplate(nx=4, nz=2, n_prism=3, n_tet=2, width=0.2), 3,
                                 ty.umesh.flatplate_bcs())):
        md = ty.preprocess(raw, dim, bcs)
        out[name] = (ty.Grid(md), md)
    return out


def states(n, mach, rng):
    """Random primitive states; velocities of random direction at up to `mach`."""
    rho, p = np.exp(rng.uniform(-1, 1, n)), np.exp(rng.uniform(-1, 1, n))
    d = rng.standard_normal((3, n))
    u = d / np.linalg.norm(d, axis=0) * rng.uniform(0, mach, n) * np.sqrt(1.4 * p / rho)
    return np.vstack([rho, p, u])


def fluxes(g, q, **spat):
    out = []
    for mode in ("exact", "fast"):
        g.set_spat(mode=mode, **spat)
        g.set_prim(q)
        g.integration_grid(1.0)
        out.append(g.debug("flux"))
    return out


def close(exact, fast):
    for rows in ([0], [1], [2, 3, 4]):
        e, f = exact[rows], fast[rows]
        assert np.isfinite(e).all()
        assert np.abs(e - f).max() <= 1e-12 * np.abs(e).max(), rows


@pytest.mark.parametrize("scheme,eps", [("ROE", 0.1), ("ROE", 0.0), ("ROE", 1.5), ("HLLC", 0.1), ("HLLCB", 0.1), ("HLLCK", 0.1),
                                        ("RUSANOV", 0.1)])
@pytest.mark.parametrize("mach", [0.05, 0.9, 3.0])
def test_inviscid(grids, scheme, eps, mach):
    g, md = grids["tet"]
    q = states(md.ncell, mach, np.random.default_rng(3))
    close(*fluxes(g, q, scheme=scheme, highres="NONE", limiter="NONE", entropy_fix=eps))


@pytest.mark.parametrize("grad", ["CELL-AVERAGE", "FULL"])
@pytest.mark.parametrize("law,nu", [("KINEMATIC-CONSTANT", 0.3), ("SUTHERLAND", 0.0)])
def test_viscous(grids, grad, law, nu):
    g, md = grids["plate"]
    q = states(md.ncell, 0.9, np.random.default_rng(4))
    if law == "SUTHERLAND":  # temperatures around 300 K, so that the viscous part is not lost in the flux
        q[0], q[1] = q[0] * 1e-6, q[1] * 1e-6 * 287.14 * 300.0
        q[2:] *= np.sqrt(287.14 * 300.0)
    close(*fluxes(g, q, scheme="HLLC", highres="NONE", limiter="NONE", dissipative_flux=grad, viscosity=law, kin_visc=nu,
                  rgas=287.14, prandtl=0.72, farfield=tuple(q[:, 0])))
