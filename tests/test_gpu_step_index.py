"""The step index of runs of several steps, which goes from one step to the
next on the device: a run gives the state and the CFL of the same steps called
one by one, wherever it starts (a call at or below step 0 takes the index after
the previous step's, step 1 is step 1) and whatever the context ran before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 3])
@pytest.mark.parametrize("ts0,nsteps,before", [
    (1, 4, 0), (1, 4, 3), (5, 3, 0), (0, 4, 0), (0, 4, 5), (-2, 6, 0), (-2, 6, 7), (-3, 2, 4),
])
def test_run_is_its_steps_one_by_one(precision, ts0, nsteps, before):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("index", 32, 8, False, 1, 0.5, subits=2, ramp=64, CFL=400.0)
    mesh = Mesh.from_grid(wl.grid(), order=1)
    fp = wl.params()
    out = []
    for whole in (True, False, None):
        s = capi.Solver.from_mesh(mesh, fp, device=0)
        s.set_precision(precision)
        s.set_state(mesh.initial_state(fp))
        for ts in range(1, before + 1):
            s.solve(ts)
        if whole:
            s.run(ts0, nsteps)
        elif whole is None:
            s.converge(ts0, nsteps, 1e-30, chunk=nsteps, check=False)
        else:
            for ts in range(ts0, ts0 + nsteps):
                s.solve(ts)
        out.append((s.get("Q"), s.get("cfl")))
        assert s.status() == 0
        s.close()
    for Q, cfl in out[1:]:
        assert np.array_equal(out[0][1], cfl)
        assert np.isfinite(Q).all() and np.array_equal(out[0][0], Q)
