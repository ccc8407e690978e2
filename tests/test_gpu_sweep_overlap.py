"""Sweep launches that start ahead of their predecessor's end: whole chunks of
steps replayed from a graph (every launch right behind the last) against the
oracle's steps, bit for bit; also where the run converges inside the chunk and
the launches left do nothing."""
import numpy as np
import pytest

from cases import chunk_order, ndiff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 3])
@pytest.mark.parametrize("nc,nr,order,subits,pairs,drop", [
    (8, 3, 1, 1, 1, 1e-30),     # one sweep: every first launch follows the assembly
    (64, 16, 1, 3, 1, 1e-30),
    (64, 16, 3, 2, 0, 1e-30),
    (128, 32, 3, 4, 1, 1e-30),
    (64, 16, 1, 3, 1, 0.9),     # converges inside the chunk
])
def test_chunk_of_steps_bitwise(mode, nc, nr, order, subits, pairs, drop):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    from oracle import port
    wl = workloads.Workload("overlap", nc, nr, order == 3, order, 0.8 if order == 3 else 0.5,
                            subits=subits)
    mesh = Mesh.from_grid(wl.grid(), order=order)
    fp = wl.params()
    Q0 = mesh.initial_state(fp)
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    og.set("Q", Q0)
    p = port.params_from_flow(fp)
    gpu = capi.Solver.from_mesh(mesh, fp, device=0)
    gpu.set_precision(mode)
    perm = None
    if mode == 3:
        gpu.set_sweep_pairs(bool(pairs))
        starts, _ = gpu.chunk_starts()
        perm, _ = chunk_order(og["ia"], og["ja"], starts)
    nn = mesh.sizes["nn"]
    gpu.set_state(Q0)
    steps, _, _ = gpu.converge(1, 12, drop, chunk=12, check=False)
    assert 1 <= steps <= 12
    for ts in range(1, steps + 1):
        if mode == 3:
            og.solve_mixed_order(p, ts, perm)
        else:
            og.solve_mixed(p, ts)
    for name in ("Q", "dQ"):
        a, b = og[name][4:4 * (nn + 1)], gpu.get(name)[4:4 * (nn + 1)]
        assert np.isfinite(b).all() and ndiff(a, b) == 0, name
    assert gpu.status() == 0
    gpu.close()
