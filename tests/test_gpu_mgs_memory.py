"""Typhon's GMRES with its vector in memory (beyond 16 entries per thread), where the grid shrinks as the
columns' sums take more shared memory, and with a second cycle after it, against the oracle's
sequential modified Gram-Schmidt.

Tolerance: the update's relative L2 per variable, 1e-9 (dot products of 1e6 terms in another order,
amplified by the condition of the least-squares problem).
"""
import numpy as np
import pytest

import oracle_py as op

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


# 31^3 x 5 cells, 744,775 unknowns: four blocks per SM up to 26 vectors, three to 36, two to 55, then one
@pytest.mark.parametrize("nkrylov,cycles", [(30, 2), (64, 1)])
def test_vector_in_memory(ty, nkrylov, cycles):
    from typhon_gb300 import cases
    w = cases.FFBOX
    ff, ln, n = w["freestream"], w["length"], 31
    raw = ty.gen_tet_box(n, ln, jitter=w["jitter"], seed=w["seed"])
    fams = ("IMIN", "IMAX", "JMIN", "JMAX", "KMIN", "KMAX")
    md = cases.make_ffbox(n)
    om = op.Mesh.from_raw(raw).build(3, [(f, op.BC_FARFIELD, "", (0.0, 0.0, 0.0)) for f in fams])
    q = cases.perturbed_freestream(md.cell_centre, ff, (ln / 2,) * 3)
    q = q * (1.0 + 0.01 * np.random.default_rng(n).standard_normal(q.shape))
    nci = md.ncell_int
    g = ty.Grid(md)
    g.set_spat("RUSANOV", "NONE", "NONE", mode="exact", farfield=ff)
    s = op.Solver(om, op.SCH_RUSANOV, op.HRES_NONE, op.LIM_NONE, farfield=ff)
    g.set_prim(q)
    U0 = g.get_cons()
    full = np.ones((5, md.ncell))
    full[:, :nci] = U0
    s.set_cons(full)
    # CFL 200: the cycles end far above the residual's rounding; the inner test is never met
    st = g.implicit_step(200.0, "GMRES", nkrylov=nkrylov, max_it=cycles - 1, inv_res=1e-14, local_dt=True)
    info, restarts, _ = s.implicit_step(200.0, local_dt=True, nkrylov=nkrylov, max_it=cycles - 1, inv_res=1e-14)
    assert st["restarts"] == restarts
    assert st["matvecs"] >= nkrylov * cycles
    du, dv = g.get_cons() - U0, s.get("cons")[:, :nci] - U0
    for rows in ([0], [1], [2, 3, 4]):
        assert np.linalg.norm(du[rows] - dv[rows]) < 1e-9 * np.linalg.norm(dv[rows]), rows
    g.close()
