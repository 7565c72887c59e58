"""The persistent conjugate-gradient kernel of heat conduction on every size of its dispatch (block
of 128, 256 and 512 threads, 1 to 12 cells per thread in registers, vectors in memory beyond), at
a fixed number of iterations, against the same preconditioned iteration in numpy on the
assembled matrix; and a solve of more iterations than one launch runs.

Tolerance: 25 iterations of a system with a modest condition number amplify rounding (1e-16) by
at most about 1e5 in the direction vectors: 1e-10 relative L2 of the update.
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


def setup(ty, n, sigma=0.5):
    from typhon_gb300 import umesh
    md = ty.preprocess(umesh.gen_kuhn_box(n, 1.0), 3, [(f, umesh.BC_WALL, "", (0.0, 0.0, 0.0)) for f in
                                                       ("IMIN", "IMAX", "JMIN", "JMAX", "KMIN", "KMAX")])
    rng = np.random.default_rng(n)
    kind, val = np.zeros(md.nface, np.int32), np.zeros(md.nface)
    b = np.arange(md.nface_int, md.nface)
    kind[b] = np.where(np.abs(md.face_centre[b, 0] - 0.5) > 0.4999, 1, 2)
    val[b] = np.where(kind[b] == 1, md.face_centre[b, 0], 0.0)
    g = ty.Grid(md)
    g.set_spat("HLLC", mode="fast")
    g.kdif_setup(np.exp(sigma * rng.standard_normal(md.ncell_int)), kind, val, flux="FULL", heat_capacity=1.3)
    T0 = rng.uniform(0.0, 1.0, md.ncell_int)
    g.kdif_set_temperature(T0)
    return md, g, T0


def matrix(md, g):
    """(diagonal, off-diagonal entries of the interior faces, cells) of the symmetrised matrix."""
    return g.kdif_get("diag"), g.kdif_get("jac")[:md.nface_int], md.fc1[:md.nface_int], md.fc2[:md.nface_int]


def product(A, x):
    d, a, c1, c2 = A
    n = len(x)
    return d * x + np.bincount(c1, a * x[c2], n) + np.bincount(c2, a * x[c1], n)


# cells 6 n^3: 128 threads (n <= 14), 256 (<= 18), 512 x 1, 2, 4, 6, 8, 10, 12 cells, in memory
@pytest.mark.parametrize("n", [3, 17, 22, 29, 36, 42, 46, 50, 53, 56])
@pytest.mark.parametrize("solver", ["CG"])
def test_fixed_iterations(ty, n, solver):
    its, dt = 25, 1e-3
    md, g, T0 = setup(ty, n)
    st = g.kdif_implicit_step(dt, solver, tol=1e-300, max_it=its)
    assert st["iterations"] == its
    x = (g.kdif_temperature() - T0) * 1.3
    A, b = matrix(md, g), g.kdif_get("balance")
    y, r = np.zeros_like(b), b.copy()
    z = r / A[0]
    p, rz = z.copy(), r @ z
    for _ in range(its):
        q = product(A, p)
        al = rz / (p @ q)
        y += al * p
        r -= al * q
        z = r / A[0]
        rz, old = r @ z, rz
        p = z + rz / old * p
    assert np.linalg.norm(x - y) < 1e-10 * np.linalg.norm(y)
    assert abs(st["rel_res"] - np.linalg.norm(r) / np.linalg.norm(b)) < 1e-8 * st["rel_res"]
    g.close()


@pytest.mark.parametrize("solver", ["CG", "CG-MIXED"])
def test_more_iterations_than_a_launch(ty, solver):
    md, g, T0 = setup(ty, 12, sigma=4.0)
    st = g.kdif_implicit_step(1e3, solver, tol=1e-10, max_it=20000)
    assert st["iterations"] > 1000 and st["rel_res"] < 1e-10
    x = (g.kdif_temperature() - T0) * 1.3
    A, b = matrix(md, g), g.kdif_get("balance")
    # the recurrence's residual drifts from the true one by rounding times the iterations
    assert np.linalg.norm(b - product(A, x)) < 1e-7 * np.linalg.norm(b)
    g.close()


def test_zero_right_hand_side(ty):
    md, g, T0 = setup(ty, 3)
    md2, g2, _ = setup(ty, 3)
    kind, val = np.zeros(md2.nface, np.int32), np.zeros(md2.nface)
    kind[md2.nface_int:] = 2
    g2.kdif_setup(np.ones(md2.ncell_int), kind, val, flux="FULL", heat_capacity=1.0)
    g2.kdif_set_temperature(np.full(md2.ncell_int, 0.5))
    st = g2.kdif_implicit_step(1e-3, "CG", tol=1e-12)
    assert st["iterations"] == 0 and st["rel_res"] == 0.0
    assert np.array_equal(g2.kdif_temperature(), np.full(md2.ncell_int, 0.5))
