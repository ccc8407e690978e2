"""The mode 3 sweep's tiles (two or four lanes a row by the mean width of a
level, padded levels, the CTA shapes) against the oracle's sweep in the same
row order: iterates bit for bit."""
import numpy as np
import pytest

from cases import chunk_order, ndiff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,nr,order,rows,levels,ring,pairs", [
    (512, 128, 3, 0, 0, 64, 1),    # 34 rows a level: two lanes a row
    (512, 128, 1, 0, 64, 32, 1),   # wider still, 64 levels a chunk
    (512, 128, 1, 2048, 24, 16, 0),
    (400, 100, 1, 0, 0, 64, 1),    # 29 rows a level: four lanes a row
    (64, 16, 1, 0, 1, 64, 1),      # chunks of a single level, a few rows each
    (32, 8, 3, 7, 3, 16, 1),       # chunks smaller than a tile
])
def test_sweep_tiles_bitwise(nc, nr, order, rows, levels, ring, pairs):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    from oracle import port
    wl = workloads.Workload("tiles", nc, nr, order == 3, order, 0.8 if order == 3 else 0.5,
                            subits=3)
    mesh = Mesh.from_grid(wl.grid(), order=order)
    fp = wl.params()
    Q0 = mesh.initial_state(fp)
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    og.set("Q", Q0)
    p = port.params_from_flow(fp)
    gpu = capi.Solver.from_mesh(mesh, fp, device=0)
    gpu.set_chunk(rows, levels)
    gpu.set_precision(3)
    gpu.set_sweep_ring(ring)
    gpu.set_sweep_pairs(bool(pairs))
    gpu.set_state(Q0)
    starts, _ = gpu.chunk_starts()
    perm, _ = chunk_order(og["ia"], og["ja"], starts)
    nn = mesh.sizes["nn"]
    for ts in (1, 2):
        og.solve_mixed_order(p, ts, perm)
        gpu.solve(ts)
        for name in ("Q", "dQ"):
            a, b = og[name][4:4 * (nn + 1)], gpu.get(name)[4:4 * (nn + 1)]
            assert np.isfinite(b).all() and ndiff(a, b) == 0, (name, ts)
    assert gpu.status() == 0
    gpu.close()
