"""The flexible GMRES' FP64 basis sweeps on vectors around one and two tiles of 480 rows (basis sizes up to
16) and of 256 rows (beyond), restarted so that every basis size up to the restart is used: each
converges to the direct solution of the assembled system, 1e-8 relative (a 1e-12 residual times a
condition number below 1e3)."""
import numpy as np
import pytest

import test_gpu_sweeps as sweeps

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


# unknowns 5 x cells: 475, 480, 495, 955, 960, 975
@pytest.mark.parametrize("ni,nj", [(5, 19), (8, 12), (9, 11), (1, 191), (12, 16), (13, 15)])
@pytest.mark.parametrize("nkrylov", [7, 16, 18])
def test_tiles(ty, ni, nj, nkrylov):
    kind = "quad"
    if ni == 1:  # a prime number of cells: a strip three nodes wide would share faces, walls do not
        md = ty.preprocess(ty.gen_grid2d(ni, nj, 0.02, 1.0, kind), 2,
                           [(f, ty.umesh.BC_FARFIELD, "", (0.0, 0.0, 0.0)) for f in ("IMIN", "IMAX", "JMIN", "JMAX")])
    else:
        md = ty.preprocess(ty.gen_grid2d(ni, nj, 1.0, 1.0, kind, jitter=0.1, seed=1), 2, ty.periodic_box_bcs((1.0, 1.0)))
    assert md.ncell_int == ni * nj
    g = sweeps.grid(ty, md, "fast")
    U0 = g.get_cons()
    st = g.implicit_step(5.0, "FGMRES", nkrylov=nkrylov, max_it=400, inv_res=1e-12, local_dt=True)
    assert st["lin_res"] <= 1e-12
    du = np.linalg.solve(sweeps.dense(md, g), g.implicit_get("rhs").reshape(-1))
    got = (g.get_cons() - U0).T.reshape(-1)
    assert np.linalg.norm(got - du) < 1e-8 * np.linalg.norm(du)
    g.close()
