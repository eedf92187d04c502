"""A solid whose bricks would share too many nodes four ways (its layers take
several bricks each) is sent back to its assembled K before any brick is built
(GPU).

The first solve of an operator may launch the layers, their order and the count
of shared nodes on top of what every later solve launches, and the transposed K.
"""
import numpy as np
import pytest

from solvix_b200 import abi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(30, 30, 30), (74, 74, 4)])
def test_compact_solid_builds_no_bricks(ctx, size):
    lib = abi.load()
    flat = workloads.cantilever_c3d8(*size, lx=0.1 * size[0], ly=0.1 * size[1],
                                     lz=0.1 * size[2], seed=5)
    op = ctx.assemble(flat)

    def solve():
        n = lib.svx_launch_count()
        u, it, res, _ = op.solve()
        return u, it, res, lib.svx_launch_count() - n

    u0, it0, res, first = solve()
    u1, it1, _, later = solve()
    assert res <= 1e-10 and it0 == it1
    np.testing.assert_array_equal(u0, u1)
    assert first - later <= 4
    op.free()
