"""The flexible GMRES' kernels at the sizes where they can go wrong: basis sweeps fed by bulk copies
(vectors of odd length, below and across one tile of 256 rows, more tiles than stages; odd and
even basis sizes up to the largest restart) and the staged block mat-vec (cell counts around its
blocks, 3 to 6 faces per cell), in FP64 and with FP32 blocks, against a dense direct solve.

The mat-vec is compared with the blocks read back (1e-13 of the largest entry: five products of
up to seven blocks).  A full-length solve (as many vectors as unknowns allow, INV_RES 1e-12) must
reach the direct solution of the assembled system: 1e-8 relative (1e-12 residual times a condition
number below 1e3).
"""
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


def make(ty, kind, n):
    if kind == "tri":
        return ty.preprocess(ty.gen_grid2d(n, n, 1.0, 1.0, "tri", jitter=0.1, seed=1), 2, ty.periodic_box_bcs((1.0, 1.0)))
    if kind == "quad":
        return ty.preprocess(ty.gen_grid2d(n, n + 1, 1.0, 1.0, "quad", jitter=0.1, seed=1), 2, ty.periodic_box_bcs((1.0, 1.0)))
    return ty.preprocess(ty.umesh.gen_flatplate(nx=n, nz=2, n_prism=3, n_tet=2, width=0.2), 3, ty.umesh.flatplate_bcs())


def grid(ty, md, mode):
    rng = np.random.default_rng(2)
    x = md.cell_centre
    q = np.stack([1 + 0.1 * np.sin(6 * x[:, 0]), 0.7 + 0.1 * np.cos(6 * x[:, 1]), 0.3 + 0.1 * np.sin(6 * x[:, 1]),
                  0.1 * np.cos(6 * x[:, 0]), 0.0 * x[:, 0]]) * (1 + 0.01 * rng.standard_normal((5, md.ncell)))
    g = ty.Grid(md)
    g.set_spat("RUSANOV", "NONE", "NONE", mode=mode, farfield=(1.0, 0.7, 0.3, 0.0, 0.0))
    g.set_prim(q)
    return g


def dense(md, g):
    """The assembled matrix from the blocks of the last FP64 step."""
    n = md.ncell_int
    A = np.zeros((n, 5, n, 5))
    i = np.arange(n)
    A[i, :, i, :] = g.implicit_get("diag")
    c1, c2 = md.fc1[:md.nface_int], md.fc2[:md.nface_int]
    for f, (u, l) in enumerate(zip(g.implicit_get("upper"), g.implicit_get("lower"))):
        A[c1[f], :, c2[f], :] += u
        A[c2[f], :, c1[f], :] += l
    return A.reshape(5 * n, 5 * n)


# unknowns 5 x cells: 90, 245, 265 (odd, around 256), 840, and cells 18 .. 168 around the mat-vec's 32 and 128
@pytest.mark.parametrize("kind,n", [("tri", 3), ("quad", 7), ("quad", 2), ("tri", 6), ("plate", 3), ("quad", 12)])
@pytest.mark.parametrize("mode", ["fast", "exact"])
def test_matvec_and_full_solve(ty, kind, n, mode):
    md = make(ty, kind, n)
    g = grid(ty, md, mode)
    U0 = g.get_cons()
    st = g.implicit_step(5.0, "FGMRES", nkrylov=32, max_it=200, inv_res=1e-12, local_dt=True)
    A, b = dense(md, g), g.implicit_get("rhs").reshape(-1)
    x = np.random.default_rng(0).standard_normal(len(b))
    y = g.implicit_matvec(x.reshape(-1, 5)).reshape(-1)
    assert np.abs(y - A @ x).max() < 1e-13 * np.abs(A).max() * np.abs(x).max() * 35
    assert st["lin_res"] <= 1e-12
    du = np.linalg.solve(A, b)
    got = (g.get_cons() - U0).T.reshape(-1)
    assert np.linalg.norm(got - du) < 1e-8 * np.linalg.norm(du)
    # the FP32 blocks converge the FP64 residual of their own system: near the FP64 update
    for precision in ("mixed-fp64ortho", "mixed"):
        h = grid(ty, md, mode)
        h.implicit_step(5.0, "FGMRES", nkrylov=17, max_it=40, inv_res=1e-5, local_dt=True, precision=precision)
        got = (h.get_cons() - U0).T.reshape(-1)
        assert np.linalg.norm(got - du) < 1e-3 * np.linalg.norm(du)
        h.close()
    g.close()


# basis sizes 1 .. 32 of one cycle on a vector of several tiles per block (odd length: 5 x 46,305)
def test_long_vectors_against_short_restarts(ty):
    from typhon_gb300 import cases
    md = cases.make_ffbox(21)
    ff = cases.FFBOX["freestream"]
    q = cases.perturbed_freestream(md.cell_centre, ff, (3.0, 3.0, 3.0))
    out = []
    for nk, cycles in ((32, 40), (9, 40)):
        g = ty.Grid(md)
        g.set_spat("RUSANOV", "NONE", "NONE", mode="fast", farfield=ff)
        g.set_prim(q)
        U0 = g.get_cons()
        st = g.implicit_step(10.0, "FGMRES", nkrylov=nk, max_it=cycles, inv_res=1e-9, local_dt=True)
        assert st["lin_res"] <= 1e-9
        out.append(g.get_cons() - U0)
        g.close()
    assert np.linalg.norm(out[0] - out[1]) < 1e-6 * np.linalg.norm(out[0])
