"""The pattern and the assembled values bit for bit against the oracle where a
node has as many elements as the list kernels hold in registers, one more,
and many more: sectors about one node (plates: 8 held) or one edge (solids:
16 held), beside nodes of few elements in the same warp."""
import numpy as np
import pytest

from oracle import oracle
from solvix_b200.marshal import FlatModel
from solvix_b200.model import ElemKind

pytestmark = pytest.mark.gpu


def ring(sectors, solid, triangles=False):
    """`sectors` kites (centre, rim k, outer k, rim k + 1) about the centre, as
    quads, as triangles without the outer node, or extruded into hexes."""
    t = 2 * np.pi * np.arange(sectors) / sectors
    h = t + np.pi / sectors
    flat = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(t), np.sin(t)], 1),
                           1.6 * np.stack([np.cos(h), np.sin(h)], 1)])
    n = flat.shape[0]
    k = np.arange(sectors)
    quad = np.stack([0 * k, 1 + k, 1 + sectors + k, 1 + (k + 1) % sectors], 1)
    layers = 2 if solid else 1
    xyz = np.concatenate([np.column_stack([flat, np.full(n, float(z))]) for z in range(layers)])
    if solid:
        conn, kind = np.concatenate([quad, quad + n], 1), ElemKind.C3d8
    elif triangles:
        conn, kind = quad[:, [0, 1, 3]], ElemKind.Cps3
    else:
        conn, kind = quad, ElemKind.Cps4
    used, conn = np.unique(conn, return_inverse=True)
    xyz = xyz[used]
    conn = conn.reshape(sectors, -1)
    ndof = 3 if solid else 2
    f = np.zeros(xyz.shape[0] * ndof)
    f[-1] = 1.0
    return FlatModel(xyz=xyz, kind=np.full(sectors, int(kind)),
                     conn_ptr=np.arange(sectors + 1) * conn.shape[1], conn=conn.ravel(),
                     youngs=np.full(sectors, 10.0), poisson=np.full(sectors, 0.3),
                     thickness=1.0, ndof=ndof, fixed_row=np.arange(2 * ndof), f=f)


@pytest.mark.parametrize("shape", ["triangles", "quads", "hexes"])
@pytest.mark.parametrize("sectors", [5, 8, 9, 16, 17, 45])
def test_pattern_of_many_elements_about_a_node(ctx, shape, sectors):
    m = ring(sectors, shape == "hexes", shape == "triangles")
    op = ctx.assemble(m, keep_original=True)
    rp, ci, v = op.csr(which=1)
    oracle.set_sort_mode(1)
    k = oracle.assemble(m)
    oracle.set_sort_mode(0)
    assert np.array_equal(rp, k.row_ptr)
    assert np.array_equal(ci.astype(np.int64), k.col_idx)
    want = np.asarray(k.vals)
    assert np.all((v.view(np.int64) == want.view(np.int64)) | ((v == 0) & (want == 0)))
