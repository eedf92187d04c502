"""Algorithmic bytes of the PCG kernels, the numerators of their rooflines.

On the assembled K the PCG path is HBM-bound, so its roofline figures divide
the bytes a kernel must move (not the bytes ncu sees it move) by its measured
duration.  The element-by-element form of C3D8 models keeps its constants and
vectors on the chip; its figure is the FP64 operations of its elements.
K is stored in node blocks (a node's ndof rows over its sorted neighbours):
one 4-byte column index per ndof x ndof block, and per node one row-block
offset and one adjacency offset (8 bytes each).
"""
from __future__ import annotations


def spmv_node_bytes(n: int, nnz: int, ndof: int, n_nodes: int, value_bytes: int = 8) -> int:
    """One node-block SpMV with p.Kp (spmv_node_dot): K values, one column
    index per block, adj_ptr and node_base, p gathered once, q written and
    p read for the dot (the vectors are FP64)."""
    return int(value_bytes * nnz + 4 * nnz // (ndof * ndof) + 16 * (n_nodes + 1) + 24 * n)


def pcg_iteration_bytes(n: int, nnz: int, ndof: int, n_nodes: int) -> int:
    """One FP64 PCG iteration: the node-block SpMV with p.Kp, then the u/r
    update (u r/w, p, r r/w, q, inv_diag) and the p update (p r/w, r,
    inv_diag)."""
    return spmv_node_bytes(n, nnz, ndof, n_nodes) + 8 * n * 11


# FP64 operations of one C3D8 element and iteration (an addition or a
# multiplication each; what the Gauss points share is counted once): modes of p
# 81, gradients of x and p 132, per Gauss point cofactors 27, scaled Lame
# constants 2, H 45, stresses 16, pull-back 45 and sums 24 (of eight points, two
# of which only start the sums, 18 less), the two planes joined 39, nodal
# forces 78, p.f 39.
HEX_ELEMENT_FLOPS = 81 + 132 + 8 * (27 + 2 + 45 + 16 + 45 + 24) - 2 * 18 + 39 + 78 + 39
# of a node: 21 additions of its elements' forces, u, r, z and p, r.r and r.z
HEX_NODE_FLOPS = 21 + 3 * (2 + 2 + 1 + 2 + 2 + 2)


def hex_iteration_flops(n_elem: int, n_nodes: int) -> int:
    """One FP64 PCG iteration of a C3D8 model, element by element."""
    return HEX_ELEMENT_FLOPS * n_elem + HEX_NODE_FLOPS * n_nodes
