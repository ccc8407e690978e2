"""Matrices with rows of more than eight off-diagonal blocks, which the FP64
sweep by bands of rows does not take: the row-by-row sweep over the whole GPU,
in its second pass over a row's blocks too, and the precision form's sweeps,
against the oracle bit for bit.  The meshes are O-grids with edges flipped
towards a few nodes until those have 9 to 20 neighbours."""
import dataclasses

import numpy as np
import pytest

from cases import ndiff


def flip_towards(grid, hubs):
    """The grid with edges opposite to each node of `hubs` (1-based node ->
    neighbours wanted) flipped to end there, where the two triangles form a
    strictly convex quadrilateral."""
    x = np.asarray(grid.x)
    tris = [list(map(int, t)) for t in grid.tris]

    def area(a, b, c):
        u, v = x[b - 1] - x[a - 1], x[c - 1] - x[a - 1]
        return u[0] * v[1] - u[1] * v[0]

    for v, want in hubs.items():
        while True:
            own = [i for i, t in enumerate(tris) if v in t]
            ring = {n for i in own for n in tris[i]} - {v}
            if len(ring) >= want:
                break
            best = None
            for i in own:
                k = tris[i].index(v)
                a, b = tris[i][(k + 1) % 3], tris[i][(k + 2) % 3]
                for j, t in enumerate(tris):
                    if j == i or a not in t or b not in t:
                        continue
                    c = next(n for n in t if n not in (a, b))
                    q = min(area(v, a, c), area(v, c, b)) / (area(v, a, b) + area(b, a, c))
                    if c not in ring and (best is None or q > best[0]):
                        best = (q, i, j, [v, a, c], [v, c, b])
            if best is None or best[0] < 0.02:
                break
            _, i, j, tris[i], tris[j] = best
    return dataclasses.replace(grid, tris=np.asarray(tris, dtype=np.asarray(grid.tris).dtype))


def wide_mesh(order, reorder=1, nc=40, nr=16):
    from flowgpu import workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("wide", nc, nr, False, order, 0.5)
    mid = (nr // 2) * nc
    hubs = {mid + 5: 9, mid + 12: 12, mid + nc + 20: 16, mid - 2 * nc + 30: 20}
    mesh = Mesh.from_grid(flip_towards(wl.grid(), hubs), order=order, reorder=reorder)
    return mesh, wl.params()


def test_the_meshes_have_wide_rows():
    """Rows on both sides of 8 and of 12 off-diagonal blocks, and some past
    16; the closed control volumes of a valid mesh."""
    from cases import closure_leak
    for order in (1, 3):
        mesh, _ = wide_mesh(order)
        ia = mesh.array("ia")
        rows = np.diff(ia[1:mesh.sizes["nn"] + 2]) - 1
        assert rows.max() > 16 and (rows == 9).any() and (rows == 12).any() and (rows == 8).any()
        assert closure_leak(mesh).max() < 1e-12


def _pair(order, mode, reorder=1, **params):
    from flowgpu import capi
    from oracle import port
    mesh, fp = wide_mesh(order, reorder)
    fp = dataclasses.replace(fp, **params)
    Q0 = mesh.initial_state(fp)
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    og.set("Q", Q0)
    gpu = capi.Solver.from_mesh(mesh, fp, device=0)
    if mode:
        gpu.set_precision(mode)
    gpu.set_state(Q0)
    return mesh, og, port.params_from_flow(fp), gpu


@pytest.mark.gpu
@pytest.mark.parametrize("reorder", [0, 1])
@pytest.mark.parametrize("order,subits", [(1, 2), (1, 3), (3, 2), (3, 1)])
def test_fp64_steps_bitwise(order, subits, reorder):
    mesh, og, p, gpu = _pair(order, 0, reorder, subits=subits)
    nn = mesh.sizes["nn"]
    for ts in range(1, 5):
        og.solve(p, ts)
        gpu.solve(ts)
        for name in ("Q", "dQ", "R"):
            a, b = og[name][4:4 * (nn + 1)], gpu.get(name)[4:4 * (nn + 1)]
            assert np.isfinite(b).all() and ndiff(a, b) == 0, (name, ts)
    # set to the precision it has, a context takes the same sweep
    gpu.set_precision(0)
    og.solve(p, 5)
    gpu.solve(5)
    assert ndiff(og["Q"][4:], gpu.get("Q")[4:]) == 0
    assert gpu.status() == 0
    gpu.close()


@pytest.mark.gpu
@pytest.mark.parametrize("subits,kind", [(1, "plain"), (2, "zeros"), (3, "extreme"), (4, "nan")])
def test_fp64_linear_solve_bitwise(subits, kind):
    """Zero and tiny right-hand sides and pivots of 1e-200 to 1e200 leave the
    range in which the solve divides by reciprocals; a NaN travels downstream
    of its row."""
    mesh, og, p, gpu = _pair(1, 0, subits=subits)
    nn = mesh.sizes["nn"]
    ia = mesh.array("ia")
    rng = np.random.Generator(np.random.PCG64(11))
    lhs = 0.1 * rng.uniform(-1.0, 1.0, (int(ia[nn + 1]), 4, 4))
    lhs[ia[2:nn + 2] - 1] += np.eye(4) * rng.uniform(2.0, 6.0, (nn, 1, 1))
    rhs = rng.standard_normal((nn + 1, 4))
    if kind == "zeros":
        rhs[rng.integers(1, nn + 1, nn // 2)] = 0.0
        rhs[rng.integers(1, nn + 1, nn // 4), 2] = -0.0
    if kind == "extreme":
        rows = rng.integers(0, nn, nn // 8)
        for i, f in zip(rows, 10.0 ** rng.uniform(-200.0, 200.0, len(rows))):
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


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("order,subits", [(1, 3), (3, 2)])
def test_precision_form_steps_bitwise(order, subits, mode):
    """A lane holds the first 12 blocks of a colour sweep's row in registers;
    the rest of a wider row, and the ordered sweep's second pass."""
    mesh, og, p, gpu = _pair(order, mode, subits=subits)
    nn = mesh.sizes["nn"]
    for ts in range(1, 5):
        og.solve_mixed(p, ts, ordered=(mode == 2))
        gpu.solve(ts)
        for name in ("Q", "dQ"):
            a, b = og[name][4:4 * (nn + 1)], gpu.get(name)[4:4 * (nn + 1)]
            assert np.isfinite(b).all() and ndiff(a, b) == 0, (name, ts)
    assert gpu.status() == 0
    gpu.close()


@pytest.mark.gpu
def test_chunked_sweeps_refuse_wide_rows():
    from flowgpu import capi
    mesh, fp = wide_mesh(1)
    s = capi.Solver.from_mesh(mesh, fp, device=0)
    with pytest.raises(capi.FlowError):
        s.set_precision(3)
    s.close()
