"""Per-kernel timing counts every kernel class of a step, the boundary edges'
among them although they otherwise run in the flux launch, and does not change
the step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,jacobian,boundary,assemble", [
    (0, 0, 5, 5), (1, 0, 5, 5), (3, 0, 5, 5), (3, 2, 5, 5),
    (3, 1, 5, 0),  # the faces' kernel forms and sums the interior faces itself
])
def test_every_class_is_counted(precision, jacobian, boundary, assemble):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("classes", 64, 16, False, 1, 0.5)
    mesh = Mesh.from_grid(wl.grid(), order=1)
    fp = wl.params()
    out, launches = [], []
    for timed in (False, True):
        s = capi.Solver.from_mesh(mesh, fp, device=0)
        s.set_precision(precision)
        if jacobian:
            s.set_jacobian(jacobian)
        s.set_state(mesh.initial_state(fp))
        s.set_timing(timed)
        n = s.launch_count()
        s.run(1, 5)
        launches.append(s.launch_count() - n)
        kt = s.kernel_times()
        if timed:
            assert kt["boundary"][0] == boundary and kt["boundary"][1] > 0.0
            assert kt["assemble"][0] == assemble
            assert kt["node_prepare"][0] == 5 and kt["subedge_flux"][0] == 5
            assert kt["sweep"][0] == 10 and kt["sweep"][1] > 0.0
        else:
            assert all(c == 0 for c, _ in kt.values())
        out.append(s.get("Q"))
        assert s.status() == 0
        s.close()
    assert np.array_equal(out[0], out[1])
    assert launches[1] - launches[0] == (0 if jacobian == 1 else 5)
