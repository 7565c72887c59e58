"""The fast mode's implicit blocks (Newton-Raphson quotients and roots, Sutherland's law as
x sqrt x) against the exact mode's on random states of the viscous plate, whose boundary kinds
fold into the left block.  Tolerance: 1e-12 of the largest entry (about a hundred FP64 operations
whose terms are at most a few times it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["HLLC", "ROE", "RUSANOV"])
@pytest.mark.parametrize("law,nu", [("KINEMATIC-CONSTANT", 0.3), ("SUTHERLAND", 0.0)])
@pytest.mark.parametrize("mach", [0.1, 2.0])
def test_fast_equals_exact(scheme, law, nu, mach):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from typhon_gb300 import build
    build.build()
    import typhon_gb300 as ty
    md = ty.preprocess(ty.umesh.gen_flatplate(nx=4, nz=2, n_prism=3, n_tet=2, width=0.2), 3, ty.umesh.flatplate_bcs())
    rng = np.random.default_rng(5)
    n = md.ncell
    q = np.empty((5, n))
    q[0] = np.exp(rng.uniform(-0.5, 0.5, n)) * 1e-6
    q[1] = q[0] * 287.14 * rng.uniform(250.0, 400.0, n)
    d = rng.standard_normal((3, n))
    q[2:] = d / np.linalg.norm(d, axis=0) * rng.uniform(0.5, 1.0, n) * mach * np.sqrt(1.4 * q[1] / q[0])
    out = []
    for mode in ("exact", "fast"):
        g = ty.Grid(md)
        g.set_spat(scheme, "NONE", "NONE", mode=mode, dissipative_flux="CELL-AVERAGE", viscosity=law, kin_visc=nu,
                   rgas=287.14, prandtl=0.72, farfield=tuple(q[:, 0]))
        g.set_prim(q)
        g.implicit_step(1.0, inversion="FGMRES", nkrylov=4, max_it=1, inv_res=0.5)
        out.append({k: g.implicit_get(k) for k in ("jacL", "jacR", "diag", "upper", "lower")})
        g.close()
    for k, e in out[0].items():
        # rows and columns of one unit together: (rho), (rho E), (rho u)
        for r in ([0], [1], [2, 3, 4]):
            for c in ([0], [1], [2, 3, 4]):
                a, b = e[:, r][:, :, c], out[1][k][:, r][:, :, c]
                assert np.isfinite(a).all()
                assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max(), (k, r, c)
