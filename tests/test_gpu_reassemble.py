"""An operator assembled again solves with the model as it is on the device:
the element operators' constants (GPU).

svx_op_reassemble re-integrates and re-assembles from the device-resident
mesh and materials.  The element-by-element solves read constants of their
own instead of K, so those have to be formed again as well: by the kernels
that the first solve after an assembly launches beside those of any other
solve of the same operator (one for bricks, two for the graph form).
"""
import os

import numpy as np
import pytest

from solvix_b200 import Context, abi, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["brick", "graph"])
def form(request):
    """A context of either element-by-element form, and its constants' kernels."""
    env = {"SVX_HEX_MIN_NODES": "0", "SVX_BRICK_MAX_ELEMS": "288"}
    if request.param == "graph":
        env["SVX_BRICK_MAX_ELEMS"] = "1"
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    c = Context(0)
    yield c, 1 if request.param == "brick" else 2
    c.close()
    for k, v in old.items():
        os.environ.pop(k, None) if v is None else os.environ.__setitem__(k, v)


def test_constants_follow_a_reassembly(form):
    ctx, constants = form
    lib = abi.load()
    op = ctx.assemble(workloads.cantilever_c3d8(24, 4, 4, lx=1.2, ly=0.2, lz=0.2, seed=11))

    def solve():
        n = lib.svx_launch_count()
        u, it, *_ = op.solve()
        return u, it, lib.svx_launch_count() - n

    u0, it0, _ = solve()  # builds the operator
    u1, it1, plain = solve()
    op.reassemble()
    u2, it2, again = solve()
    assert it0 == it1 == it2
    assert again == plain + constants
    np.testing.assert_array_equal(u0, u1)
    np.testing.assert_array_equal(u0, u2)
    assert solve()[2] == plain  # and only once
    op.free()
