"""Chunks of steps that really are replayed from a graph (the first chunk of a
call is launched step by step, so a call needs several), and a run that
converges inside a replayed chunk: the launches left do nothing, the step index
and the CFL stay those of the last step, and the context goes on from there.
Against the oracle, bit for bit."""
import dataclasses

import numpy as np
import pytest

from cases import chunk_order, ndiff

pytestmark = pytest.mark.gpu


def _oracle_run(mesh, fp, mode, perm, nsteps):
    """The oracle after each step: (||R_rho||, Q, dQ, cfl)."""
    from oracle import port
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    og.set("Q", mesh.initial_state(fp))
    p = port.params_from_flow(fp)
    out = []
    for ts in range(1, nsteps + 1):
        if mode == 3:
            og.solve_mixed_order(p, ts, perm)
        elif mode:
            og.solve_mixed(p, ts)
        else:
            og.solve(p, ts)
        R = og["R"].reshape(-1, 4)[1:, 0]
        cfl = 1. + (1. * (ts - 1)) / (1. * fp.ramp) * (fp.CFL - 1.) if ts < fp.ramp else fp.CFL
        out.append((float(np.sqrt((R * R).sum())), og["Q"].copy(), og["dQ"].copy(), cfl))
    return out


@pytest.mark.parametrize("mode", [0, 1, 3])
@pytest.mark.parametrize("chunk,subits", [(4, 4), (4, 2), (3, 4), (5, 3)])
def test_stop_inside_a_replayed_chunk(mode, chunk, subits):
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("stop", 64, 16, True, 3, 0.8, subits=subits)
    mesh = Mesh.from_grid(wl.grid(), order=3)
    fp = wl.params()
    gpu = capi.Solver.from_mesh(mesh, fp, device=0)
    perm = None
    if mode:
        gpu.set_precision(mode)
    if mode == 3:
        perm, _ = chunk_order(mesh.array("ia"), mesh.array("ja"), gpu.chunk_starts()[0])
    nsteps = 4 * chunk
    want = _oracle_run(mesh, fp, mode, perm, nsteps + 2)
    nn = mesh.sizes["nn"]

    def check(ts):
        _, Q, dQ, cfl = want[ts - 1]
        assert ndiff(Q[4:], gpu.get("Q")[4:]) == 0, ts
        assert ndiff(dQ[4:4 * (nn + 1)], gpu.get("dQ")[4:]) == 0, ts
        assert gpu.get("cfl")[0] == cfl, ts

    # all four chunks, three of them replayed
    gpu.set_state(mesh.initial_state(fp))
    steps, _, _ = gpu.converge(1, nsteps, 1e-30, chunk=chunk, check=False)
    assert steps == nsteps
    check(nsteps)
    assert gpu.capture_fallbacks() == 0

    # a drop that step `last`, not the end of its chunk, is the first to reach
    r = [w[0] for w in want]
    last = next(s for s in range(chunk + 1, nsteps) if s % chunk and r[s - 1] < 0.98 * min(r[:s - 1]))
    drop = 0.5 * (r[last - 1] + min(r[:last - 1])) / r[0]
    gpu.set_state(mesh.initial_state(fp))
    steps, _, _ = gpu.converge(1, nsteps, drop, chunk=chunk)
    assert steps == last
    check(last)
    for ts in (last + 1, last + 2):
        gpu.solve(ts)
        check(ts)
    assert gpu.status() == 0
    gpu.close()
