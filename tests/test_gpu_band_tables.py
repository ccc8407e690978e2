"""When a context lays out the tables of the FP64 sweep by bands: with its first
FP64 solve, once, from its own arena where it has one and only while room is
left; never for single stages or the precision form.  The results do not depend
on it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(nc=64, nr=16, order=1):
    from flowgpu import workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("bands", nc, nr, False, order, 0.5, subits=3)
    return Mesh.from_grid(wl.grid(), order=order), wl.params()


def _in_arena(arena, mesh, fp):
    """A Solver carved from an arena (flow_create_in)."""
    import ctypes as C
    from flowgpu import capi
    s = capi.Solver.__new__(capi.Solver)
    s.L, s._keep, s.params, s.sizes = capi.load(), None, fp, mesh.sizes
    s.p = capi.params_struct(fp)
    st = C.c_int(0)
    s.ctx = s.L.flow_create_in(arena.h, C.byref(mesh.view), C.byref(s.p), C.byref(st))
    assert s.ctx, st.value
    return s


def _bytes(s):
    return s.L.flow_ctx_device_bytes(s.ctx)


def _uses_bands(s):
    """The self-test's launches: 3, and 4 more where the sweeps go by bands."""
    from flowgpu import capi
    n = s.launch_count()
    assert s.selftest_sweep_timeout(64) == capi.ERR_SWEEP_TIMEOUT
    return s.launch_count() - n == 7


def _steps(s, mesh, fp):
    s.set_state(mesh.initial_state(fp))
    for ts in (1, 2, 3):
        s.solve(ts)
    return s.get("Q")


def test_only_fp64_solves_lay_the_tables_out():
    from flowgpu import capi
    mesh, fp = _case()
    s = capi.Solver.from_mesh(mesh, fp, device=0)
    n0 = _bytes(s)
    s.set_state(mesh.initial_state(fp))
    s.set_precision(0)
    s.build_matrix(1)
    s.reconstruct(1)
    s.residuals(1, 1)
    assert _bytes(s) == n0
    s.linear_solve()
    n1 = _bytes(s)
    rows = mesh.sizes["nn"]
    assert 32 * rows <= n1 - n0 <= 128 * rows
    s.linear_solve()
    s.set_precision(0)
    s.linear_solve()
    assert _bytes(s) == n1
    s.close()
    s = capi.Solver.from_mesh(mesh, fp, device=0)
    s.set_precision(3)
    n3 = _bytes(s)
    s.set_state(mesh.initial_state(fp))
    s.solve(1)  # takes the history of a step's norms
    assert _bytes(s) - n3 <= 4096
    s.close()


@pytest.mark.parametrize("room", ["much", "none", "exact"])
def test_arena_contexts_take_the_same_steps(room):
    from flowgpu import capi
    mesh, fp = _case()
    s = capi.Solver.from_mesh(mesh, fp, device=0)
    need = _bytes(s) + 4096  # and the history of a step's norms
    want = _steps(s, mesh, fp)
    tables = _bytes(s) - need
    assert _uses_bands(s) and tables > 0
    s.close()
    size = {"much": 1 << 30, "none": need, "exact": 2 * need + tables - 4096}[room]
    arena = capi.Arena(size)
    s = _in_arena(arena, mesh, fp)
    free = arena.free_bytes()
    s.set_precision(0)
    assert arena.free_bytes() == free
    assert np.array_equal(_steps(s, mesh, fp), want)
    assert _uses_bands(s) == (room == "much")
    assert arena.free_bytes() >= free - 4096 or room == "much"
    if room != "none":  # what the context may yet carve still fits
        s.save_state()
        s.set_precision(1)
        s.set_precision(0)
    assert s.status() == 0
    s.close()
    arena.close()


def test_refused_matrix_keeps_the_row_sweep():
    from flowgpu import capi
    from test_gpu_wide_rows import wide_mesh
    mesh, fp = wide_mesh(1)
    s = capi.Solver.from_mesh(mesh, fp, device=0)
    s.set_state(mesh.initial_state(fp))
    s.solve(1)
    n = _bytes(s)
    assert not _uses_bands(s)
    s.set_precision(0)
    s.solve(2)
    assert _bytes(s) == n and s.status() == 0
    s.close()


def test_first_solve_as_replayed_chunks():
    """The tables are there before a chunk of steps is captured, also when the
    context comes back from the precision form."""
    from flowgpu import capi
    mesh, fp = _case(128, 32)
    out = []
    for detour in (False, True):
        s = capi.Solver.from_mesh(mesh, fp, device=0)
        if detour:
            s.set_precision(3)
            s.set_state(mesh.initial_state(fp))
            s.converge(1, 12, 1e-30, chunk=4, check=False)
            s.set_precision(0)
        s.set_state(mesh.initial_state(fp))
        s.converge(1, 12, 1e-30, chunk=4, check=False)
        out.append(s.get("Q"))
        assert _uses_bands(s) and s.status() == 0
        s.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("room", ["much", "tight"])
def test_fp64_requests_through_the_server(room):
    """FP64 requests admitted from host threads beside running ones take the
    steps that they take alone, with the tables and where they find no room."""
    import concurrent.futures as cf
    from flowgpu import capi
    cases = [_case(64, 16), _case(96, 24), _case(40, 10), _case(128, 32)]
    alone, need = [], 0
    for mesh, fp in cases:
        s = capi.Solver.from_mesh(mesh, fp, device=0)
        need += _bytes(s) + (1 << 16)
        s.set_state(mesh.initial_state(fp))
        steps, _, _ = s.converge(1, 96, 1e-10, chunk=16, check=False)
        alone.append((steps, s.get("Q")))
        s.close()
    arena = capi.Arena((1 << 30) if room == "much" else need)
    srv = capi.Server(arena, chunk=16, max_slots=8)

    def admit(i):
        mesh, fp = cases[i]
        while True:
            slot = srv.submit(mesh, fp, mesh.initial_state(fp), precision=0, drop=1e-10,
                              max_steps=96, tag=i)
            if slot is not None:
                return slot

    got = {}
    with cf.ThreadPoolExecutor(max_workers=4) as ex:
        futs = [ex.submit(admit, i) for i in range(len(cases))]
        while len(got) < len(cases):
            for c in srv.progress(wait_us=500):
                q, _ = srv.result(c["slot"])
                srv.release(c["slot"])
                got[c["tag"]] = (c["steps"], q)
            for f in futs:
                if f.done():
                    f.result()
    for i, (steps, q) in enumerate(alone):
        assert got[i][0] == steps
        assert np.array_equal(q[4:], got[i][1][4:])
    srv.close()
    arena.close()
