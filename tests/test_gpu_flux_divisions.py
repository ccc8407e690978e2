"""The face flux where its divisions by reciprocals hand over to the divisions
themselves (velocities of zero, minus zero or far below the fast range), against
the oracle bit for bit: residual, Jacobian blocks and update."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["zero", "minus zero", "tiny", "all at rest", "mixed"])
@pytest.mark.parametrize("nc,nr,order", [(24, 9, 1), (34, 11, 3)])
def test_step_bitwise(nc, nr, order, kind):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    from oracle import port
    wl = workloads.Workload("div", nc, nr, order == 3, order, 0.5, alpha=0.0, subits=2)
    mesh = Mesh.from_grid(wl.grid(), order=order)
    fp = wl.params()
    nn = mesh.sizes["nn"]
    rng = np.random.Generator(np.random.PCG64(11))
    Q0 = np.array(mesh.initial_state(fp)).reshape(-1, 4)
    q = Q0[1:nn + 1]
    q[:, 0] *= rng.uniform(0.9, 1.1, nn)
    pick = rng.integers(0, 5, nn)
    vals = {"zero": 0.0, "minus zero": -0.0, "tiny": 1e-40}
    if kind in vals:
        q[pick == 0, 1] = vals[kind]
        q[pick <= 1, 2] = vals[kind]
    elif kind == "all at rest":
        q[:, 1:3] = 0.0
    else:
        for i, v in enumerate((0.0, -0.0, 1e-40, -1e-300)):
            q[pick == i, 1 + i % 2] = v
    Q0 = np.ascontiguousarray(Q0.reshape(-1))
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    og.set("Q", Q0)
    p = port.params_from_flow(fp)
    gpu = capi.Solver.from_mesh(mesh, fp, device=0)
    gpu.set_state(Q0)
    og.solve(p, 1)
    gpu.solve(1)
    nnz = int(mesh.array("ia")[nn + 1])
    for name, n in (("R", 4 * (nn + 1)), ("LHS", 16 * nnz), ("dQ", 4 * (nn + 1))):
        a, b = og[name][:n], gpu.get(name)[:n]
        assert np.array_equal(a[4:], b[4:], equal_nan=True), name
        if name == "R":
            assert np.isfinite(a[4:]).all()
    gpu.close()
