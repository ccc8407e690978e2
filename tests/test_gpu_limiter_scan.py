"""The node kernel's limiter scan (two divisions a side instead of two a face
point) against the oracle's point-by-point fold, bit for bit, in every form of
the kernel, on fields chosen for where the scan must hand over to the fold or
meets its special values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("smooth", "uniform", "ulp", "repeated", "tiny", "huge", "nan", "inf")


def _field(mesh, Q0, kind):
    rng = np.random.Generator(np.random.PCG64(FIELDS.index(kind)))
    v = mesh.view
    n = v.nn + v.nn_ghost + 1
    x = mesh.array("x").reshape(n, 2)
    Q = Q0.reshape(n, 4).copy()
    bump = np.exp(-((x - [0.3, 0.4]) ** 2).sum(axis=1))
    if kind == "smooth":
        Q *= 1.0 + 0.05 * bump[:, None] * rng.uniform(0.5, 1.0, 4)
    elif kind == "ulp":        # differences of an ulp or two: many equal ones
        Q *= 1.0 + 2.3e-16 * rng.integers(-2, 3, Q.shape)
    elif kind == "repeated":   # a few distinct values: equal decisive points
        Q *= 1.0 + 0.01 * rng.integers(0, 2, Q.shape)
    elif kind == "tiny":       # a momentum around zero, down to where FP32 underflows
        Q[:, 2] = 1e-42 * rng.standard_normal(n) * (rng.random(n) < 0.7)
        Q[:, 1] *= 1.0 + 1e-33 * rng.standard_normal(n)
    elif kind == "huge":       # a node's differences beyond FP32's range
        Q[rng.integers(1, v.nn + 1, 20), 3] = 1e200
    elif kind in ("nan", "inf"):
        Q[rng.integers(1, v.nn + 1, 12), rng.integers(0, 4, 12)] = (
            np.nan if kind == "nan" else np.inf)
    Q[0] = 0.0
    return Q.reshape(-1)


@pytest.mark.parametrize("order", [1, 3])
@pytest.mark.parametrize("kind", FIELDS)
def test_phi_bitwise(order, kind):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    from oracle import port
    wl = workloads.Workload("scan", 46, 11, order == 3, order, 0.6)
    mesh = Mesh.from_grid(wl.grid(), order=order)
    fp = wl.params()
    nn = mesh.sizes["nn"]
    Q = _field(mesh, mesh.initial_state(fp), kind)
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    og.set("Q", Q)
    og.set("nQ", Q)
    og.g.citer = 1
    p = port.params_from_flow(fp)
    with np.errstate(all="ignore"):
        (og.gradient if order == 1 else og.derivatives)()
        og.limiter(p)
    gpu = capi.Solver.from_mesh(mesh, fp, device=0)
    gpu.set_state(Q)
    names = ["phi"] + (["grad"] if order == 1 else ["point_value", "hess"])
    for variant in range(8):
        gpu.set_variants(variant, 0)
        try:
            gpu.reconstruct(1)
        except capi.FlowError:  # the state is not physical: the arrays are compared all the same
            gpu.L.flow_clear_status(gpu.ctx)
        for name in names:
            w = og[name].size // (nn + 1)
            a, b = og[name][w:w * (nn + 1)], gpu.get(name)[w:w * (nn + 1)]
            assert np.array_equal(a, b, equal_nan=True), (name, variant)
    gpu.close()
