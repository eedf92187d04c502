"""From which size solid batch members go element by element (GPU).

Below 180 nodes a large batch is faster on the assembled K, so those members
stay on it: their batch launches what it launches in a context without the
element-by-element forms, and from 180 on the bricks' build kernels as well.
"""
import os

import pytest

from solvix_b200 import Context, abi, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def on_k():
    old = os.environ.get("SVX_HEX")
    os.environ["SVX_HEX"] = "0"
    c = Context(0)
    os.environ.pop("SVX_HEX") if old is None else os.environ.__setitem__("SVX_HEX", old)
    yield c
    c.close()


@pytest.mark.parametrize("size,bricks", [((12, 2, 2), False), ((8, 3, 3), False),
                                         ((10, 3, 3), False), ((19, 2, 2), True),
                                         ((11, 3, 3), True)])
def test_members_take_bricks_from_180_nodes(ctx, on_k, size, bricks):
    lib = abi.load()
    flat = workloads.cantilever_c3d8(*size, lx=0.1 * size[0], ly=0.1 * size[1],
                                     lz=0.1 * size[2], seed=3)
    assert (flat.n_nodes >= 180) == bricks

    def launches(c):
        n = lib.svx_launch_count()
        c.solve_batch([flat, flat])
        return lib.svx_launch_count() - n

    assert (launches(ctx) > launches(on_k)) == bricks
