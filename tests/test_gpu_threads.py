"""Two handles, each driven by a thread of its own: Krylov solves whose kernels take different amounts of
shared memory at the same moment.  Every step succeeds and gives the state of the same step alone, bit
for bit (fixed grids, fixed orders)."""
import threading

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


def both(work, alone, rounds):
    """Runs work(0) and work(1) repeatedly in two threads; every result equals alone[i]."""
    errors = []

    def run(i):
        try:
            for _ in range(rounds):
                assert np.array_equal(work(i), alone[i])
        except BaseException as e:  # noqa: BLE001 - reported by the main thread
            errors.append((i, e))

    t = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not errors, errors


def test_gmres_columns(ty):
    from typhon_gb300 import cases as wl
    md, ff = wl.make_ffbox(6), wl.FFBOX["freestream"]
    q = wl.perturbed_freestream(md.cell_centre, ff, (0.5 * wl.FFBOX["length"],) * 3)[:, :md.ncell_int]
    gs = [ty.Grid(md) for _ in range(2)]
    for g in gs:
        g.set_spat("RUSANOV", mode="fast", farfield=ff)

    def work(i):
        gs[i].set_prim(q)
        gs[i].implicit_step(200.0, "GMRES", nkrylov=(60, 7)[i], max_it=(2, 12)[i], inv_res=1e-13)
        return gs[i].get_cons()

    both(work, [work(0), work(1)], 12)
    for g in gs:
        g.close()


def test_heat_lists(ty):
    from typhon_gb300 import umesh
    walls = [(f, umesh.BC_WALL, "", (0.0, 0.0, 0.0)) for f in ("IMIN", "IMAX", "JMIN", "JMAX", "KMIN", "KMAX")]
    tet = ty.preprocess(umesh.gen_kuhn_box(29, 1.0), 3, walls)  # 146,334 cells: two per thread, four faces
    tri = ty.preprocess(umesh.gen_grid2d(270, 270, 1.0, 1.0, "tri"), 2, walls[:4])  # 145,800 cells, three faces
    gs, Ts = [], []
    for md in (tet, tri):
        g = ty.Grid(md)
        g.set_spat("HLLC", mode="fast")
        kind = np.zeros(md.nface, np.int32)
        kind[md.nface_int:] = 1
        g.kdif_setup(np.ones(md.ncell_int), kind, np.zeros(md.nface), flux="COMPACT", heat_capacity=1.0)
        gs.append(g)
        Ts.append(np.random.default_rng(1).uniform(0.0, 1.0, md.ncell_int))

    def work(i):
        for _ in range(20):
            gs[i].kdif_set_temperature(Ts[i])
            gs[i].kdif_implicit_step(1e-6, "CG", tol=1e-3)
        return gs[i].kdif_temperature()

    both(work, [work(0), work(1)], 12)
    for g in gs:
        g.close()
