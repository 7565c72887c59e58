"""The cooperative Gram-Schmidt kernel of Typhon's GMRES on every size of its dispatch (1 to 16
entries of the vector per thread, the vector in memory beyond) and up to 64 Krylov vectors, and
the block mat-vec on both sides of the row form's limit: one GMRES cycle of a far-field box's
implicit step against the oracle's (sequential modified Gram-Schmidt).

Tolerance: the update's relative L2 per variable, 1e-9 (dot products of 1e4 to 1e6 terms in
another order, amplified by the condition of the least-squares problem).
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


# unknowns 25 n^3: 1, 2, 4, 8, 16 entries per thread of 152 x 256, and in memory
@pytest.mark.parametrize("n,nkrylov", [(2, 12), (11, 20), (11, 64), (14, 20), (17, 20), (22, 12), (29, 12), (31, 12)])
def test_one_cycle_against_oracle(ty, n, nkrylov):
    from typhon_gb300 import cases
    w = cases.FFBOX
    ff, ln = w["freestream"], w["length"]
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
    # an inner test that is never met, so that all nkrylov vectors are built
    st = g.implicit_step(20.0, "GMRES", nkrylov=nkrylov, max_it=0, inv_res=1e-14, local_dt=True)
    info, restarts, _ = s.implicit_step(20.0, local_dt=True, nkrylov=nkrylov, max_it=0, inv_res=1e-14)
    assert st["restarts"] == restarts
    du, dv = g.get_cons() - U0, s.get("cons")[:, :nci] - U0
    for rows in ([0], [1], [2, 3, 4]):
        assert np.linalg.norm(du[rows] - dv[rows]) < 1e-9 * np.linalg.norm(dv[rows]), rows
    g.close()
