"""The byte counts of the roofline count what a launch shares once: the face
Jacobians that flux and assembly hand over, the node states that faces and rows
gather.  Each count is set against the arrays' own sizes, taken from the mesh."""
import pytest


def _mesh(order):
    from flowgpu import workloads
    from flowgpu.prep import Mesh
    wl = workloads.Workload("rl_u", 64, 16, order == 3, order, 0.8)
    return Mesh.from_grid(wl.grid(), order=order)


def _counts(m):
    ia = m.array("ia")
    nn = m.sizes["nn"]
    return nn, m.sizes["nsubedges"], m.sizes["nbedges"], int(ia[nn + 1]) - int(ia[1])


@pytest.mark.parametrize("approx", [False, True])
@pytest.mark.parametrize("order", [1, 3])
def test_flux_counts_each_node_and_face_once(order, approx):
    from flowgpu import roofline
    m = _mesh(order)
    nn, ns, nbe, _ = _counts(m)
    written = ns * (32 + (128 if approx else 256)) + nbe * (32 + 128)
    read = ns * (8 + 32) + nbe * (16 + 24) + nn * 32
    if order == 1:
        read += ns * 32 + nn * (64 + 16)
    assert roofline.subedge_flux_bytes(m, approx=approx) == read + written
    # without the Jacobian: less its blocks and the boundary's
    assert roofline.subedge_flux_bytes(m) - roofline.subedge_flux_bytes(m, jacobian=False) == \
        ns * 256 + nbe * 128


@pytest.mark.parametrize("precision,approx", [(0, False), (1, False), (3, False), (3, True)])
def test_assembly_reads_each_jacobian_once(precision, approx):
    from flowgpu import roofline
    m = _mesh(3)
    nn, ns, nbe, nnz = _counts(m)
    faces = ns * (32 + (128 if approx else 256)) + nbe * (32 + 128)  # what the flux wrote
    lists = ns * 8 + (nnz - nn) * (4 + 16) + nbe * 4 + nn * 20
    nodes = nn * (16 + 64)
    rows = {0: nnz * 128 + nn * (128 + 32 + 32), 1: (nnz - nn) * 64 + nn * (64 + 16),
            3: (nnz - nn) * 64 + nn * (80 + 16)}[precision]
    assert roofline.assemble_bytes(m, precision, approx) == faces + lists + nodes + rows
