"""An implicit step waits for its own stream only: not for work that the caller has on the legacy
default stream, which the handle's non-blocking stream does not meet."""
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


@pytest.mark.parametrize("inversion", ["GMRES", "FGMRES"])
def test_step_does_not_wait_for_the_default_stream(ty, inversion):
    import torch
    from typhon_gb300 import cases as wl
    md, ff = wl.make_ffbox(6), wl.FFBOX["freestream"]
    g = ty.Grid(md)
    g.set_spat("RUSANOV", mode="fast", farfield=ff)
    q = wl.perturbed_freestream(md.cell_centre, ff, (0.5 * wl.FFBOX["length"],) * 3)[:, :md.ncell_int]

    def step():
        return g.implicit_step(10.0, inversion, nkrylov=10, max_it=2, inv_res=1e-3)

    g.set_prim(q)
    step()  # allocations, and a kernel's first use, wait for the whole device
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.default_stream()):
        torch.cuda._sleep(int(1e9))  # half a second; the step takes milliseconds
        ev = torch.cuda.Event()
        ev.record()
    step()
    assert not ev.query()
    torch.cuda.synchronize()
    g.close()
