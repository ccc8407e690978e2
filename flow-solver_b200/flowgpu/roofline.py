"""Algorithmic (compulsory) DRAM bytes per launch of the main kernels.

Each figure counts every array element a launch must read or write once:
per-node records, per-face records, incidence lists, stencils, and the
outputs.  What several threads of a launch read is counted once: a node's
state however many faces or rows gather it, a face's Jacobian blocks although
its two nodes read each for their diagonal and their off-diagonal blocks (the
other reads can be cache hits).  The achieved bandwidth of a launch is
these bytes over its measured duration; DRAM traffic measured by ncu well
above them would mean re-reads.
"""
from __future__ import annotations

import numpy as np


def _sizes(mesh) -> dict:
    v = mesh.view
    out = {"nn": v.nn, "ns": v.nsubedges, "ne": v.nedges, "nbe": v.nbedges, "stencil": 0}
    if mesh.order == 3:
        m = np.ctypeslib.as_array(v.svd_m, shape=(v.nn + 1,))
        out["stencil"] = int(m[1:].sum())
    nnz = int(np.ctypeslib.as_array(v.ia, shape=(v.nn + 2,))[v.nn + 1])
    out["nnz"] = nnz
    return out


def node_prepare_bytes(mesh) -> int:
    """k_node_prepare4: wave-speed sum and dt, the k=1 gradient or the k=2
    derivatives (x = V S^-1 U^T b over the node's stencil) and point value,
    and the Venkatakrishnan limiter over every face point.

    per node   read  nQ 32, x 16, cv_area 8, three incidence pointers 12
                     (k=2: the record of S, 1/S, moments and V^T 352, stencil pointer 4)
               write dt 8, phi 64 (k=1: grad 64; k=2: derivatives 160, point values 32)
    per subedge      two incidence entries 8, normal/length 32,
                     face point offsets 32 (k=1) or 3 Gauss points 48 (k=2)
    per edge         two neighbour entries 8 (k=1: two incidence entries 8, LSQ weights 32)
    per bedge        incidence entry 4, normal/length 24
    per stencil entry (k=2) index 4, weight 8, the row of U's first 5 columns 40
    """
    z = _sizes(mesh)
    k2 = mesh.order == 3
    per_node = 32 + 16 + 8 + 12 + 8 + 64 + ((352 + 4 + 160 + 32) if k2 else 64)
    per_sub = 8 + 32 + (48 if k2 else 32)
    per_edge = 8 + (0 if k2 else 8 + 32)
    per_bedge = 4 + 24
    return int(z["nn"] * per_node + z["ns"] * per_sub + z["ne"] * per_edge +
               z["nbe"] * per_bedge + z["stencil"] * 52)


def colour_sweep_bytes(mesh) -> int:
    """One whole multicolour FP32 sweep (all colour launches): per row the
    row record 16, right-hand side 32 (FP64), LU factors 64, the iterate read
    and written 32; per off-diagonal block its column 4 and the block 64
    (FP32)."""
    z = _sizes(mesh)
    offd = z["nnz"] - z["nn"]
    return int(z["nn"] * (16 + 32 + 64 + 32) + offd * (4 + 64))


def ordered_sweep_bytes(mesh) -> int:
    """One FP64 ordered sweep (k_sweep_bands): per block 128 B of LHS and
    4 B of column index, per row RHS, LU of the diagonal, dQ read and write
    (132 B per block + 96 B per row, the diagonal block counted as a block).
    What this kernel reads besides is left out, since the sweep does not need
    it: the pivots' reciprocals (32 B a row, they follow from the factors) and
    the rest of its 32-byte slots (a row's columns are counted as above)."""
    z = _sizes(mesh)
    return int(132 * z["nnz"] + 96 * z["nn"])


def chunk_sweep_bytes(mesh) -> int:
    """One whole chunked FP32 sweep (precision mode 3, all colour launches):
    per row its factors and right-hand side 80, window positions and row word
    20, its iterate read through the chunk's window and written back (16 +
    16); per off-diagonal block its FP32 values 64."""
    z = _sizes(mesh)
    offd = z["nnz"] - z["nn"]
    return int(z["nn"] * (80 + 20 + 32) + offd * 64)


def subedge_flux_bytes(mesh, jacobian: bool = True, approx: bool = False) -> int:
    """k_subedge_flux: per node its state 32 read (k=1 reconstruction: its
    gradient 64 and two limiter values 16); per subedge its end nodes 8 and
    normal/length 32 read (k=1: the face-point offsets 32), the flux 32
    written and, with the Jacobian, dF/dqL and dF/dqR: 256 (FP64) or, for the
    approximate Jacobian of the precision form, 128 (FP32).  The boundary
    edges in the launch's first blocks, per edge: its record 16 and normal 24
    read, its flux 32 and, with the Jacobian, its block 128 written."""
    z = _sizes(mesh)
    jac = (128 if approx else 256) if jacobian else 0
    k1 = mesh.order != 3
    return int(z["nn"] * (32 + (64 + 16 if k1 else 0)) +
               z["ns"] * (8 + 32 + (32 if k1 else 0) + 32 + jac) +
               z["nbe"] * (16 + 24 + 32 + (128 if jacobian else 0)))


def assemble_bytes(mesh, precision: int = 3, approx: bool = False) -> int:
    """k_assemble4: per subedge its two incidence entries 8, its flux 32 and
    its two Jacobian blocks 2J read; per off-diagonal block its column 4 and
    subedge pair 16; per boundary edge its incidence entry 4, flux 32 and block
    128; per node dt, cv_area 16 and five list pointers 20 read, R and RHS 64
    and the cleared iterate 16 (FP32) or 32 written, and its row: its FP32
    blocks 64 a block, factors and right-hand side 80 (mode 3; without the
    right-hand side, 64, modes 1 and 2), or FP64 blocks 128 a block, LU factors
    128 and the pivots' reciprocals 32 (mode 0).  J = 128 (FP64) or 64 (the
    approximate Jacobian's FP32 blocks)."""
    z = _sizes(mesh)
    offd = z["nnz"] - z["nn"]
    J = 64 if approx else 128
    if precision == 0:
        rows = 128 * z["nnz"] + (128 + 32 + 32) * z["nn"]
    else:
        rows = 64 * offd + ((80 if precision == 3 else 64) + 16) * z["nn"]
    return int(z["ns"] * (8 + 32 + 2 * J) + offd * (4 + 16) + z["nbe"] * (4 + 32 + 128) +
               z["nn"] * (16 + 20 + 64) + rows)


def faces_assemble_bytes(mesh) -> int:
    """k_faces_assemble (precision form, approximate Jacobian): per subedge its
    two incidence entries and block slots 16, end nodes 8 and normal/length 32
    read (k=1: the face-point offsets 32); per node its state 32 (k=1: its
    gradient 64 and two limiter values 16), dt and cv_area 16 read, R and RHS
    64, the cleared iterate 16 and its row's factors and right-hand side 80
    written; per off-diagonal block 64; per boundary edge its flux and block
    160 read."""
    z = _sizes(mesh)
    k1 = mesh.order != 3
    offd = z["nnz"] - z["nn"]
    return int(z["ns"] * (16 + 8 + 32 + (32 if k1 else 0)) +
               z["nn"] * (32 + (64 + 16 if k1 else 0) + 16 + 64 + 16 + 80) + offd * 64 +
               z["nbe"] * 160)
