"""Device memory of a batch of solids on bricks: what a member takes does not
grow with the largest member beside it (GPU).

Each size of batch runs in a context of its own, whose device memory is what
the process gained by it.  The bricks of 600 members of 180 nodes and one
large member are to fit what the two take apart; room by the largest brick
(2,800 node slots of 140 bytes instead of 608) took 290 KB a member more.
"""
import pytest
import torch

from solvix_b200 import Context, workloads

pytestmark = pytest.mark.gpu


def test_small_members_beside_a_large_one(ctx):
    small = workloads.cantilever_c3d8(19, 2, 2, lx=1.9, ly=0.2, lz=0.2, seed=1)
    large = workloads.cantilever_c3d8(60, 16, 16, lx=6.0, ly=1.6, lz=1.6, seed=2)

    def used(flats):
        free0 = torch.cuda.mem_get_info()[0]
        with Context(0) as c:
            _, st = c.solve_batch(flats)
            assert st["not_converged"] == 0
            return free0 - torch.cuda.mem_get_info()[0]

    used([small, large])  # streams and kernels are loaded
    apart = used([small] * 600) + used([large])
    together = used([small] * 600 + [large])
    assert together - apart < 600 * 100e3
