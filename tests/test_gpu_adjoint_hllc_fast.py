"""The fast mode's reverse of HLLC on random states from Mach 0 to 3, which take its four wave
patterns and both choices of either wave speed, against the exact mode's reverse (checked on
the host against dual numbers); first order, where no limiter stands between.

Tolerance: 1e-12 of the largest entry, and of the vector in L2 (two hundred FP64 operations whose
terms are at most a few times the result; an ulp is 1.1e-16).  Second order with van Albada,
where a sign of a b near 0 may fall between the modes' roundings of the gradient: random cell
states keep it away from 0, so 1e-10 in L2 (the slopes' quotients amplify by about a hundred).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("highres,limiter,tol", [("NONE", "NONE", 1e-12), ("MUSCL", "ALBADA", 1e-10),
                                                 ("MUSCL-UNS", "ALBADA", 1e-10)])
@pytest.mark.parametrize("mach", [0.05, 0.9, 3.0])
@pytest.mark.parametrize("n", [2, 4])
def test_fast_equals_exact(highres, limiter, tol, mach, n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from typhon_gb300 import build
    build.build()
    import typhon_gb300 as ty
    from typhon_gb300 import adjoint
    md = ty.preprocess(ty.gen_tet_box(n, 1.0, jitter=0.05, seed=2), 3, ty.periodic_box_bcs((1.0,) * 3))
    rng = np.random.default_rng(7)
    nci = md.ncell_int
    q = np.empty((5, nci))
    q[0], q[1] = np.exp(rng.uniform(-0.2, 0.2, nci)), np.exp(rng.uniform(-0.2, 0.2, nci))
    d = rng.standard_normal((3, 1)) + 0.1 * rng.standard_normal((3, nci))
    q[2:] = d / np.linalg.norm(d, axis=0) * rng.uniform(0.9, 1.1, nci) * mach * np.sqrt(1.4 * q[1] / q[0])
    U = torch.tensor(ty.prim_to_cons(q), device="cuda")
    lam = torch.tensor(rng.standard_normal((5, nci)), device="cuda")
    out = []
    for mode in ("exact", "fast"):
        g = ty.Grid(md)
        g.set_spat("HLLC", highres, limiter, mode=mode)
        out.append(adjoint.Stepper(g, "RK2").vjp(U, 1e-3, lam).cpu().numpy())
        g.close()
    exact, fast = out
    assert np.isfinite(exact).all()
    assert np.linalg.norm(fast - exact) <= tol * np.linalg.norm(exact)
    if highres == "NONE":
        assert np.abs(fast - exact).max() <= tol * np.abs(exact).max()
