"""Conduction systems (one dof a node) on the device against the oracle, at
the sizes where the assembly's groups of four nodes a warp and the PCG's
slices of 32 rows can go wrong: node counts about their multiples, more and
fewer slices than blocks, plates of triangles and quads together, a quad
that repeats a node beside others in its warp, a node of a large degree
(rows wider than a slice takes), several launches of one solve.

Bar: the assembled values are summed in the same element order, the PCG's
reductions are not, so the two temperatures are each off by the condition
of the scaled system times the tolerance asked of both: about L^2 x 1e-13
for L nodes along the longer side (or around the fan).  2 L^2 x 1e-13, and
never less than the 1e-10 of the other conduction solves."""
import numpy as np
import pytest

from oracle import oracle
from solvix_b200.marshal import ThermalModel
from solvix_b200.model import ElemKind

pytestmark = pytest.mark.gpu

TOL = 1e-13


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def plate(nx, ny, collapsed=False):
    """nx x ny cells, every third one split into two triangles."""
    rng = np.random.Generator(np.random.PCG64(nx * 1000 + ny))
    xs, ys = np.meshgrid(np.arange(nx + 1.0), np.arange(ny + 1.0))
    xyz = np.zeros(((nx + 1) * (ny + 1), 3))
    xyz[:, 0], xyz[:, 1] = xs.ravel(), ys.ravel()
    inner = (xyz[:, 0] > 0) & (xyz[:, 0] < nx) & (xyz[:, 1] > 0) & (xyz[:, 1] < ny)
    xyz[inner, :2] += rng.uniform(-0.15, 0.15, (int(inner.sum()), 2))
    conn, kind, ptr = [], [], [0]
    for j in range(ny):
        for i in range(nx):
            a = j * (nx + 1) + i
            b, c, d = a + 1, a + nx + 2, a + nx + 1
            if (i + j) % 3 == 1:
                cells = [[a, b, c], [a, c, d]]
            elif collapsed and (i + j) % 3 == 2:
                cells = [[a, b, c, c], [a, c, d]]
            else:
                cells = [[a, b, c, d]]
            for q in cells:
                conn += q
                ptr.append(len(conn))
                kind.append(int(ElemKind.Cps4 if len(q) == 4 else ElemKind.Cps3))
    return finish(xyz, kind, ptr, conn, 0.5)


def block(nx, ny, nz):
    def nid(i, j, k):
        return (k * (ny + 1) + j) * (nx + 1) + i
    xyz = np.array([(i, j, k) for k in range(nz + 1) for j in range(ny + 1)
                    for i in range(nx + 1)], float)
    conn = [q for k in range(nz) for j in range(ny) for i in range(nx)
            for q in (nid(i, j, k), nid(i + 1, j, k), nid(i + 1, j + 1, k), nid(i, j + 1, k),
                      nid(i, j, k + 1), nid(i + 1, j, k + 1), nid(i + 1, j + 1, k + 1),
                      nid(i, j + 1, k + 1))]
    ne = nx * ny * nz
    return finish(xyz, [int(ElemKind.C3d8)] * ne, np.arange(ne + 1) * 8, conn, 1.0)


def fan(spokes):
    """One node with `spokes` triangles about it: a row of spokes + 1."""
    t = np.linspace(0.0, 2 * np.pi, spokes, endpoint=False)
    xyz = np.zeros((spokes + 1, 3))
    xyz[1:, 0], xyz[1:, 1] = np.cos(t), np.sin(t)
    conn = [q for k in range(spokes) for q in (0, 1 + k, 1 + (k + 1) % spokes)]
    return finish(xyz, [int(ElemKind.Cps3)] * spokes, np.arange(spokes + 1) * 3, conn, 0.5)


def finish(xyz, kind, ptr, conn, thickness):
    ends = np.concatenate([np.flatnonzero(xyz[:, 0] == xyz[:, 0].min()),
                           np.flatnonzero(xyz[:, 0] == xyz[:, 0].max())])
    value = np.where(xyz[ends, 0] == xyz[:, 0].min(), 20.0, 80.0)
    return ThermalModel(xyz, kind, ptr, conn, 12.0, thickness, source=3.0, temp_node=ends,
                        temp_value=value)


CASES = {
    "one_quad": (2, lambda: plate(1, 1)),
    "30_nodes": (10, lambda: plate(9, 2)),
    "32_nodes": (8, lambda: plate(7, 3)),
    "33_nodes": (11, lambda: plate(10, 2)),
    "slices_one_a_block": (74, lambda: plate(73, 63)),  # 4,736 nodes: 148 slices
    "slices_one_more": (82, lambda: plate(57, 81)),     # 4,756 nodes: 149 slices
    "collapsed_quads": (14, lambda: plate(13, 11, collapsed=True)),
    "fan_of_31": (31, lambda: fan(31)),                 # the widest row of a slice
    "fan_of_32": (32, lambda: fan(32)),                 # one wider
    "fan_of_900": (900, lambda: fan(900)),              # a warp's four nodes need more room
    "cube_of_8": (3, lambda: block(2, 2, 2)),
    "block": (41, lambda: block(40, 6, 5)),
    "many_launches": (1501, lambda: plate(1500, 1)),    # more iterations than one launch runs
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_conduction_matches_oracle(ctx, name):
    length, make = CASES[name]
    m = make()
    got = ctx.solve_thermal(m, tol=TOL)
    want = oracle.solve_thermal(m, tol=TOL)
    assert rel(got[0], want[0]) <= max(1e-10, 2 * length**2 * TOL)
