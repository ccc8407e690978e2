"""The sweeps' wait for a dependency level: it gives every lane of the waiting
warp one answer, and gives up after its tries on a level that nothing
completes.  The self-test checks both on the device before it lets an ordered
sweep's polls run out."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_spin", [1, 64, 4096])
@pytest.mark.parametrize("nc,nr", [(8, 3), (64, 16)])
def test_every_wait_of_the_self_test_reports(nc, nr, max_spin):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("levelwait", nc, nr, False, 1, 0.5)
    mesh = Mesh.from_grid(wl.grid(), order=1)
    s = capi.Solver.from_mesh(mesh, wl.params(), device=0)
    for _ in range(8):
        assert s.selftest_sweep_timeout(max_spin=max_spin) == capi.ERR_SWEEP_TIMEOUT
    assert s.status() == 0
    s.close()
