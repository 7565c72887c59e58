"""The fast mode's fused cell kernel (one thread per cell and variable) against the CPU oracle on
meshes of 3, 4, 5 and 6 faces per cell, with cell counts around its blocks of 32 cells, every
limiter form, the Barth post-limiter (FP32 comparisons with an FP64 fallback) at ordinary and
extreme scales, and the ghost states it writes on periodic meshes.

Tolerance: the fast mode's envelope against the oracle, 1e-12 relative L2 per conserved variable.
"""
import numpy as np
import pytest

import oracle_py as op

pytestmark = pytest.mark.gpu

RTOL = 1e-12
HRES = {"MUSCL": op.HRES_MUSCL, "MUSCL-FAST": op.HRES_MUSCLFAST, "MUSCL-UNS": op.HRES_MUSCLUNS}
LIM = {"NONE": op.LIM_NONE, "MINMOD": op.LIM_MINMOD, "ALBADA": op.LIM_ALBADA, "VAN_LEER": op.LIM_VLEER,
       "SUPERBEE": op.LIM_SBEE, "KIM3": op.LIM_KIM3, "LIM03": op.LIM_LIM03}
POST = {"NONE": op.POSTLIM_NONE, "BARTH": op.POSTLIM_BARTH, "SUPERBARTH": op.POSTLIM_SUPERBARTH}


@pytest.fixture(scope="module")
def ty():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from typhon_gb300 import build
    build.build()
    import typhon_gb300
    return typhon_gb300


def hexa_box(ty, n):
    """n^3 hexahedra on [0, 1]^3, inner nodes jittered, boundary quadrangles marked per plane."""
    um = ty.umesh
    g = np.arange(n + 1) / n
    vt = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    ijk = np.stack(np.unravel_index(np.arange(len(vt)), (n + 1,) * 3), 1)
    inner = ((ijk > 0) & (ijk < n)).all(1)
    vt[inner] += np.random.default_rng(5).uniform(-0.1 / n, 0.1 / n, (inner.sum(), 3))
    vid = lambda i, j, k: (i * (n + 1) + j) * (n + 1) + k + 1
    I, J, K = (a.reshape(-1) for a in np.meshgrid(*(np.arange(n),) * 3, indexing="ij"))
    corner = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    hexa = np.stack([vid(I + a, J + b, K + c) for a, b, c in corner], 1).astype(np.int32)
    p, q = (a.reshape(-1) for a in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    quads, marks, nxt = [], [], 1
    for name, ax, val in (("IMIN", 0, 0), ("IMAX", 0, n), ("JMIN", 1, 0), ("JMAX", 1, n), ("KMIN", 2, 0), ("KMAX", 2, n)):
        f = []
        for a, b in ((0, 0), (1, 0), (1, 1), (0, 1)):
            t = [p + a, q + b]
            t.insert(ax, np.full_like(p, val))
            f.append(vid(*t))
        quads.append(np.stack(f, 1))
        marks.append((name, np.arange(nxt, nxt + len(p), dtype=np.int32)))
        nxt += len(p)
    quads = np.concatenate(quads).astype(np.int32)
    secs = [(um.ELEM_HEXA8, np.arange(1, len(hexa) + 1, dtype=np.int32), hexa),
            (um.ELEM_QUAD4, np.arange(1, len(quads) + 1, dtype=np.int32), quads)]
    return um.RawMesh(vtex=vt, sections=secs, marks=marks), 3, ty.periodic_box_bcs((1.0,) * 3), 6


def plate(ty, n):
    return ty.umesh.gen_flatplate(nx=n, nz=2, n_prism=3, n_tet=2, width=0.2), 3, ty.umesh.flatplate_bcs(), 5


def mesh(ty, kind, n):
    if kind == "hexa":
        return hexa_box(ty, n)
    if kind == "plate":
        return plate(ty, n)
    if kind == "tet":
        return ty.gen_tet_box(n, 1.0, jitter=0.05, seed=3), 3, ty.periodic_box_bcs((1.0,) * 3), 4
    return ty.gen_grid2d(n, n + 1, 1.0, 1.0, kind, jitter=0.1, seed=3), 2, ty.periodic_box_bcs((1.0, 1.0)), 3 if kind == "tri" else 4


def state(md, dim, scale=1.0):
    """Smooth fields with a per-cell random part; scale multiplies density and pressure."""
    rng = np.random.default_rng(11)
    x = md.cell_centre
    q = np.stack([1.0 + 0.1 * np.sin(2 * np.pi * x[:, 0]), 2.0 + 0.2 * np.cos(2 * np.pi * x[:, 1]),
                  0.5 + 0.1 * np.sin(2 * np.pi * x[:, 1]), 0.1 * np.cos(2 * np.pi * x[:, 0]),
                  0.2 * np.sin(2 * np.pi * (x[:, 0] + x[:, 2]))])
    q *= 1.0 + 0.02 * rng.standard_normal(q.shape)
    if dim == 2:
        q[4] = 0.0
    q[:2] *= scale
    return q


def check(ty, kind, n, highres, limiter, postlim="NONE", scale=1.0):
    raw, dim, bcs, nslot = mesh(ty, kind, n)
    md = ty.preprocess(raw, dim, bcs)
    q = state(md, dim, scale)
    ff = (scale, 2.0 * scale, 0.5, 0.0, 0.0)
    g = ty.Grid(md)
    assert g.info()["max_faces_per_cell"] == nslot
    # a no-slip wall's cell state needs a viscosity (0 / 0 conductivity otherwise, in both codes)
    visc = dict(dissipative_flux="CELL-AVERAGE", kin_visc=1e-3) if kind == "plate" else {}
    g.set_spat("HLLC", highres, limiter, postlim, mode="fast", farfield=ff, **visc)
    g.set_prim(q)
    om = op.Mesh.from_raw(raw).build(dim, [tuple(b) for b in bcs])
    s = op.Solver(om, op.SCH_HLLC, HRES[highres], LIM[limiter], POST[postlim], op.GRAD_LSQ, rk="RK4", cfl=0.5, farfield=ff,
                  **(dict(viscous=op.VISC_CELLAVG, visc_kin=1e-3) if visc else {}))
    s.set_prim(q)
    dt = s.timestep()
    nci = md.ncell_int
    g.integration_grid(dt)
    s.rhs(dt)
    if kind != "plate":  # the ghosts the cell kernel writes: copies of interior states
        gp, sp = g.debug("prim")[:, nci:], s.get("prim")[:, nci:]
        assert np.abs(gp - sp).max() <= 1e-14 * np.abs(sp).max()
    g.set_prim(q)
    s.set_prim(q)
    g.treelevel_rungekutta("RK4", dt)
    s.rk_step(dt)
    a, b = g.get_cons(), s.get("cons")[:, :nci]
    for rows in ([0], [1], [2, 3, 4]):
        err = np.linalg.norm(a[rows] - b[rows]) / np.linalg.norm(b[rows])
        assert err < RTOL, (rows, err)


# 31 .. 33 cells are not reachable with every kind: counts below, across and beyond one block
@pytest.mark.parametrize("kind,n", [("tri", 3), ("tri", 7), ("quad", 5), ("quad", 8), ("tet", 2), ("tet", 4), ("plate", 4),
                                    ("hexa", 3), ("hexa", 4)])
@pytest.mark.parametrize("highres,limiter", [("MUSCL", "ALBADA"), ("MUSCL-UNS", "ALBADA"), ("MUSCL-FAST", "ALBADA"),
                                             ("MUSCL-UNS", "NONE"), ("MUSCL-FAST", "LIM03")])
def test_residual_and_step(ty, kind, n, highres, limiter):
    check(ty, kind, n, highres, limiter)


@pytest.mark.parametrize("limiter", ["MINMOD", "VAN_LEER", "SUPERBEE", "KIM3", "LIM03"])
@pytest.mark.parametrize("highres", ["MUSCL", "MUSCL-UNS"])
def test_limiters(ty, highres, limiter):
    check(ty, "tet", 4, highres, limiter)


# 1e-40 and 1e40: differences outside the FP32 comparison's range take the FP64 products
@pytest.mark.parametrize("scale", [1.0, 1e-40, 1e40])
@pytest.mark.parametrize("kind,n,highres,limiter,postlim", [("tet", 4, "MUSCL-UNS", "NONE", "BARTH"),
                                                            ("hexa", 3, "MUSCL", "NONE", "SUPERBARTH"),
                                                            ("tri", 7, "MUSCL", "ALBADA", "BARTH")])
def test_barth(ty, kind, n, highres, limiter, postlim, scale):
    check(ty, kind, n, highres, limiter, postlim, scale)
