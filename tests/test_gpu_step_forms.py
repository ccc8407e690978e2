"""Every form of a step against the oracle's restatement, bit for bit: Newton
iterations, steps without a Jacobian update, start-up steps of lower order, no
limiter, no, one and odd sweeps; called one by one, as one run (a step begins
where the one before ended) and as chunks of steps replayed from a graph.  And
every variant of the node kernel, with the arrays that it writes."""
import dataclasses

import numpy as np
import pytest

from cases import chunk_order, ndiff

pytestmark = pytest.mark.gpu


def _mesh(nc, nr, order, **params):
    from flowgpu import workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("forms", nc, nr, order == 3, order, 0.8 if order == 3 else 0.5)
    mesh = Mesh.from_grid(wl.grid(), order=order)
    return mesh, dataclasses.replace(wl.params(), **params)


def _oracle(mesh, fp, mode, starts):
    """A function that takes the oracle's grid through step ts."""
    from oracle import port
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    og.set("Q", mesh.initial_state(fp))
    p = port.params_from_flow(fp)
    if mode == 0:
        return og, lambda ts: og.solve(p, ts)
    if mode == 3:
        perm, _ = chunk_order(og["ia"], og["ja"], starts)
        return og, lambda ts: og.solve_mixed_order(p, ts, perm)
    return og, lambda ts: og.solve_mixed(p, ts, ordered=(mode == 2))


def _solver(mesh, fp, mode):
    from flowgpu import capi
    s = capi.Solver.from_mesh(mesh, fp, device=0)
    s.set_precision(mode)
    s.set_state(mesh.initial_state(fp))
    return s


def _check(og, s, order, ts, names):
    nn = og.sizes["nn"]
    for name in names:
        a, b = og[name], s.get(name)
        if name == "hess":
            a, b = (v.reshape(-1, 4, 9)[1:, :, :5] for v in (a, b))
        else:
            w = 8 if name in ("phi", "grad") else 4
            a, b = a[w:], b[w:]
            if name in ("R", "dQ"):
                a, b = a[:4 * nn], b[:4 * nn]
        assert np.isfinite(b).all() and ndiff(a, b) == 0, (name, ts)


# an iteration without a Jacobian update is explicit: its rows take a CFL at
# which the oracle's run stays finite
FORMS = [
    (1, {"iter": 3, "jufreq": 2, "CFL": 0.5}),
    (3, {"iter": 3, "jufreq": 2, "CFL": 0.5}),
    (3, {"iter": 2, "jufreq": 1, "subits": 3}),
    (1, {"iter": 3, "jufreq": 5, "limit": 0, "CFL": 0.5}),  # clears phi before every iteration
    (1, {"limit": 0}),
    (3, {"limit": 0}),
    (1, {"foits": 3}),
    (3, {"foits": 3}),
    (3, {"foits": 2, "soits": 2}),
    (3, {"soits": 3, "iter": 2, "jufreq": 2, "CFL": 0.5}),
    (1, {"subits": 0}),
    (3, {"subits": 1}),
    (1, {"subits": 5}),
]


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("order,params", FORMS)
def test_step_forms_bitwise(order, params, mode):
    mesh, fp = _mesh(40, 10, order, **params)
    nsteps = 7
    one = _solver(mesh, fp, mode)
    starts = one.chunk_starts()[0] if mode == 3 else None
    og, step = _oracle(mesh, fp, mode, starts)
    for ts in range(1, nsteps + 1):
        step(ts)
        one.solve(ts)
        _check(og, one, order, ts,
               ["Q", "nQ", "pQ", "R", "dQ", "phi", "grad"] + (["hess"] if order == 3 else []))
    assert one.status() == 0
    one.close()
    for call in (lambda s: s.run(1, nsteps),
                 lambda s: s.converge(1, nsteps, 1e-30, chunk=2, check=False),
                 lambda s: s.converge(1, nsteps, 1e-30, chunk=nsteps, check=False)):
        s = _solver(mesh, fp, mode)
        call(s)
        _check(og, s, order, nsteps, ["Q", "nQ", "pQ", "R", "dQ", "phi", "grad"])
        assert s.status() == 0
        s.close()


@pytest.mark.parametrize("variant", range(8))
@pytest.mark.parametrize("nc,nr,order,params", [
    (128, 32, 1, {}),
    (128, 32, 3, {}),
    (12, 4, 3, {}),                          # 48 nodes
    (40, 10, 3, {"foits": 1, "soits": 2}),   # the first-order gradient's kernel in a k=2 context
    (40, 10, 1, {"limit": 0}),
    (40, 10, 3, {"limit": 0}),
])
def test_node_variants_bitwise(nc, nr, order, params, variant):
    mesh, fp = _mesh(nc, nr, order, **params)
    s = _solver(mesh, fp, 0)
    s.set_variants(variant, variant % 3)
    og, step = _oracle(mesh, fp, 0, None)
    for ts in range(1, 6):
        step(ts)
        s.solve(ts)
        _check(og, s, order, ts, ["Q", "R", "phi", "grad"] + (["hess"] if order == 3 else []))
        assert ndiff(og["LHS"], s.get("LHS")) == 0, ts
    assert s.status() == 0
    s.close()
