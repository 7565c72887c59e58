"""The stage kernels' launches: the three time-step slots that take turns over the steps of one
call, and the face kernel on both sides of the size at which it is launched dependently.

Steps of one call against the same number of single steps, each with the time step of a call of
its own: bit for bit in the exact mode; in the fast mode the two time steps are rounded apart by
a few ulp (about ten operations), so 1e-13 on dt and 1e-12 of the largest value on the state.
Face fluxes against the exact mode's: 1e-12 of the largest (a hundred operations).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def box(n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from typhon_gb300 import build
    build.build()
    import typhon_gb300 as ty
    md = ty.preprocess(ty.gen_tet_box(n, 1.0, jitter=0.05, seed=5), 3, ty.periodic_box_bcs((1.0,) * 3))
    return ty.Grid(md), md


def state(md, seed=6):
    rng = np.random.default_rng(seed)
    q = np.empty((5, md.ncell))
    q[0], q[1] = 1.0 + 0.1 * rng.random(md.ncell), 1.0 + 0.1 * rng.random(md.ncell)
    q[2:] = 0.3 * rng.standard_normal((3, md.ncell))
    return q


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("steps", [1, 2, 3, 4, 7])
def test_slots(mode, steps):
    g, md = box(4)
    g.set_spat(scheme="HLLC", highres="MUSCL", limiter="ALBADA", mode=mode)
    out = []
    for one_call in (True, False):
        g.set_prim(state(md))
        if one_call:
            dt = g.run_steps("RK3-SSP", 0.5, steps)
        else:
            for _ in range(steps):
                dt = g.calc_zonetimestep(0.5)
                g.treelevel_rungekutta("RK3-SSP", dt)
        out.append((dt, g.get_cons()))
    (da, a), (db, b) = out
    if mode == "exact":
        assert da == db and np.array_equal(a, b)
    else:
        assert abs(da - db) <= 1e-13 * db
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("n", [22, 24])  # 2 x 5 n^3 faces: 106,480 and 138,240 around 131,072
def test_face_kernel_sizes(n):
    g, md = box(n)
    out = []
    for mode in ("exact", "fast"):
        g.set_spat(scheme="ROE", highres="NONE", limiter="NONE", mode=mode)
        g.set_prim(state(md))
        g.integration_grid(1.0)
        out.append(g.debug("flux"))
    for rows in ([0], [1], [2, 3, 4]):
        assert np.abs(out[0][rows] - out[1][rows]).max() <= 1e-12 * np.abs(out[0][rows]).max()
