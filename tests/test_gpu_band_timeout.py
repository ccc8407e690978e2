"""The bounded waits of the FP64 sweep by bands of rows: with a band that never
runs, both directions give up, report the time-out and end, on two bands and on
more bands than run at once; the context then takes the steps of one that never
ran the test, bit for bit."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,nr,max_spin", [(64, 16, 1), (64, 16, 4096), (160, 40, 512),
                                            (640, 160, 64)])
def test_a_band_that_never_runs(nc, nr, max_spin):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("bandwait", nc, nr, False, 1, 0.5, subits=3)
    mesh = Mesh.from_grid(wl.grid(), order=1)
    fp = wl.params()
    a, b = (capi.Solver.from_mesh(mesh, fp, device=0) for _ in range(2))
    for s in (a, b):
        s.set_state(mesh.initial_state(fp))
        s.solve(1)
    # the level's wait, the row-by-row sweep, the sweep by bands both ways
    n = a.launch_count()
    t0 = time.monotonic()
    assert a.selftest_sweep_timeout(max_spin=max_spin) == capi.ERR_SWEEP_TIMEOUT
    assert time.monotonic() - t0 < 5.0
    assert a.launch_count() - n == 7
    assert a.status() == 0
    for ts in (2, 3):
        a.solve(ts)
        b.solve(ts)
        for name in ("Q", "dQ"):
            assert np.array_equal(a.get(name), b.get(name)), (name, ts)
    assert a.status() == 0 and b.status() == 0
    a.close()
    b.close()
