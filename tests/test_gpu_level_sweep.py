"""The FP64 ordered sweep by bands of rows and dependency levels against the
oracle, bit for bit: whole steps, meshes in other row numberings, and linear
solves of systems whose pivots and right-hand sides reach past the range in
which it divides by reciprocals."""
import dataclasses

import numpy as np
import pytest

from cases import ndiff

pytestmark = pytest.mark.gpu


def _renumbered(grid, numbering):
    """The grid with its nodes in random order or reversed."""
    n = grid.x.shape[0]
    perm = np.random.Generator(np.random.PCG64(5)).permutation(n) if numbering == "random" \
        else np.arange(n)[::-1]  # new index of node i
    x = np.empty_like(np.asarray(grid.x))
    x[perm] = grid.x
    bnds = [(bc, perm[np.asarray(segs) - 1] + 1) for bc, segs in grid.boundaries]
    return dataclasses.replace(grid, x=x, tris=perm[np.asarray(grid.tris) - 1] + 1,
                               boundaries=bnds)


def _setup(nc, nr, order, subits, numbering="reordered"):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    from oracle import port
    wl = workloads.Workload("levels", nc, nr, order == 3, order, 0.8 if order == 3 else 0.5,
                            subits=subits)
    if numbering == "reordered":
        mesh = Mesh.from_grid(wl.grid(), order=order)
    else:
        grid = wl.grid()
        mesh = Mesh.from_grid(grid if numbering == "natural" else _renumbered(grid, numbering),
                              order=order, reorder=0)
    fp = wl.params()
    Q0 = mesh.initial_state(fp)
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    og.set("Q", Q0)
    gpu = capi.Solver.from_mesh(mesh, fp, device=0)
    gpu.set_state(Q0)
    return mesh, og, port.params_from_flow(fp), gpu


@pytest.mark.parametrize("nc,nr,order,subits,steps", [
    (8, 3, 1, 2, 3),       # 24 nodes: levels of a row or two
    (12, 4, 3, 3, 3),      # an odd number of sweeps
    (40, 16, 1, 2, 3),     # 640 rows: one band
    (66, 17, 3, 2, 3),     # 1,122 rows: a full band and a part
    (128, 32, 1, 4, 3),
    (400, 100, 1, 2, 2),   # 60 rows a level
    (640, 160, 3, 1, 1),   # 102,400 rows: more bands than SMs
])
def test_steps_bitwise(nc, nr, order, subits, steps):
    mesh, og, p, gpu = _setup(nc, nr, order, subits)
    nn = mesh.sizes["nn"]
    for ts in range(1, steps + 1):
        og.solve(p, ts)
        gpu.solve(ts)
        for name in ("Q", "dQ", "R"):
            assert ndiff(og[name][4:4 * (nn + 1)], gpu.get(name)[4:4 * (nn + 1)]) == 0, (name, ts)
    assert gpu.status() == 0
    gpu.close()


@pytest.mark.parametrize("numbering", ["natural", "reversed", "random"])
@pytest.mark.parametrize("nc,nr,subits", [(48, 14, 3), (160, 40, 2)])
def test_numberings_bitwise(nc, nr, subits, numbering):
    """Rings a band, levels against the bands' order, and halos of thousands
    of rows that cross bands at every level."""
    mesh, og, p, gpu = _setup(nc, nr, 1, subits, numbering)
    nn = mesh.sizes["nn"]
    for ts in (1, 2):
        og.solve(p, ts)
        gpu.solve(ts)
        for name in ("Q", "dQ"):
            assert ndiff(og[name][4:4 * (nn + 1)], gpu.get(name)[4:4 * (nn + 1)]) == 0, (name, ts)
    assert gpu.status() == 0
    gpu.close()


@pytest.mark.parametrize("nc,nr,subits,kind", [
    (32, 8, 2, "plain"),
    (64, 16, 3, "zeros"),      # rows with a zero right-hand side
    (64, 16, 2, "extreme"),    # pivots and right-hand sides of 1e-200 to 1e200
    (96, 24, 4, "nan"),        # a NaN travels downstream of its row
])
def test_linear_solve_bitwise(nc, nr, subits, kind):
    mesh, og, p, gpu = _setup(nc, nr, 1, subits)
    nn = mesh.sizes["nn"]
    ia = mesh.array("ia")
    rng = np.random.Generator(np.random.PCG64(7))
    lhs = 0.2 * rng.uniform(-1.0, 1.0, (int(ia[nn + 1]), 4, 4))
    diag = ia[2:nn + 2] - 1
    lhs[diag] += np.eye(4) * rng.uniform(2.0, 6.0, (nn, 1, 1))
    rhs = rng.standard_normal((nn + 1, 4))
    if kind == "zeros":
        rhs[rng.integers(1, nn + 1, nn // 2)] = 0.0
        rhs[rng.integers(1, nn + 1, nn // 4), 2] = -0.0
    if kind == "extreme":
        rows = rng.integers(0, nn, nn // 8)
        scale = 10.0 ** rng.uniform(-200.0, 200.0, len(rows))
        for i, f in zip(rows, scale):  # the whole row, so that its solution stays ordinary
            lhs[ia[i + 1]:ia[i + 2]] *= f
            rhs[i + 1] *= f
    if kind == "nan":
        rhs[nn // 2, 1] = np.nan
    rhs[0] = 0.0
    og.set("LHS", lhs.reshape(-1))
    og.set("RHS", rhs.reshape(-1))
    og["dQ"][:] = 0.0
    gpu.set("LHS", lhs.reshape(-1))
    gpu.set("RHS", rhs.reshape(-1))
    want = og.linear_solve(p)
    got = gpu.linear_solve()
    a, b = og["dQ"][4:4 * (nn + 1)], gpu.get("dQ")[4:4 * (nn + 1)]
    assert np.array_equal(a, b, equal_nan=True)
    if kind in ("plain", "zeros"):
        assert abs(got - want) <= 1e-12 * want
    assert gpu.status() == 0
    gpu.close()
