"""The b - Ax RMS by quads of lanes: against a row-order sum in numpy over
sizes from one row to many blocks' worth, aligned and misaligned caller
arrays; summed in the reference's order it is the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(nn, seed):
    """A BCSR system of 1 to 11 blocks a row; row 0 unused."""
    rng = np.random.Generator(np.random.PCG64([seed, nn]))
    cnt = rng.integers(1, 12, nn)
    ia = np.zeros(nn + 2, dtype=np.int32)
    ia[2:] = np.cumsum(cnt)
    nnz = int(ia[nn + 1])
    ja = rng.integers(1, nn + 1, nnz).astype(np.int32)
    lhs = rng.standard_normal((nnz, 4, 4))
    rhs, x = rng.standard_normal((nn + 1, 4)), rng.standard_normal((nn + 1, 4))
    row = np.repeat(np.arange(1, nn + 1), cnt)
    ax = np.zeros((nn + 1, 4))
    np.add.at(ax, row, np.einsum("kij,kj->ki", lhs, x[ja]))
    want = np.sqrt(((rhs - ax)[1:] ** 2).sum() / nn)
    return ia, ja, lhs, rhs, x, nnz, want


@pytest.mark.parametrize("nn", [1, 2, 63, 64, 65, 75775, 75776, 75777, 262144])
@pytest.mark.parametrize("shift", [0, 1])
def test_noalloc_rms(nn, shift):
    import torch
    from flowgpu import capi
    ia, ja, lhs, rhs, x, nnz, want = _system(nn, 3)

    def dev(a):
        t = torch.zeros(a.size + shift, dtype=torch.float64, device="cuda")
        t[shift:] = torch.from_numpy(a.reshape(-1))
        return t, t.data_ptr() + 8 * shift
    keep = [torch.from_numpy(ia).cuda(), torch.from_numpy(ja).cuda()]
    bufs = [dev(a) for a in (lhs, rhs, x)]
    torch.cuda.synchronize()
    for _ in range(2):
        got = capi.linear_residual_noalloc(keep[0].data_ptr(), keep[1].data_ptr(),
                                           *[p for _, p in bufs], nn, nnz)
        # 12 terms of size about 1 a component and a sum of positive squares
        assert abs(got - want) <= 1e-13 * want
    bad = keep[1].clone()
    bad[nnz // 2] = nn + 1
    with pytest.raises(capi.FlowError):
        capi.linear_residual_noalloc(keep[0].data_ptr(), bad.data_ptr(), *[p for _, p in bufs],
                                     nn, nnz)
    got = capi.linear_residual_noalloc(keep[0].data_ptr(), keep[1].data_ptr(),
                                       *[p for _, p in bufs], nn, nnz)
    assert abs(got - want) <= 1e-13 * want


@pytest.mark.parametrize("nc,nr,scale", [(8, 3, 1.0), (64, 16, 1.0), (128, 32, 1e-16)])
def test_exact_rms_is_the_oracles(nc, nr, scale):
    """scale 1e-16: an RMS below 1e-15, which ends the sweeps early."""
    from flowgpu import capi, workloads
    from flowgpu.prep import Mesh
    from oracle import port
    wl = workloads.Workload("rms", nc, nr, False, 1, 0.5, subits=4)
    mesh = Mesh.from_grid(wl.grid(), order=1)
    fp = wl.params()
    og = port.OracleGrid(mesh.sizes, mesh.arrays())
    gpu = capi.Solver.from_mesh(mesh, fp, device=0)
    gpu.set_exact_rms(True)
    nn = mesh.sizes["nn"]
    ia = mesh.array("ia")
    rng = np.random.Generator(np.random.PCG64(5))
    lhs = 0.2 * rng.uniform(-1.0, 1.0, (int(ia[nn + 1]), 4, 4))
    lhs[ia[2:nn + 2] - 1] += 4.0 * np.eye(4)
    rhs = scale * rng.standard_normal((nn + 1, 4))
    rhs[0] = 0.0
    for s, name, a in ((s, name, a) for s in (og, gpu) for name, a in (("LHS", lhs), ("RHS", rhs))):
        s.set(name, a.reshape(-1))
    og["dQ"][:] = 0.0
    want = og.linear_solve(port.params_from_flow(fp))
    assert gpu.linear_solve() == want
    assert np.array_equal(og["dQ"][4:4 * (nn + 1)], gpu.get("dQ")[4:4 * (nn + 1)])
    gpu.close()
