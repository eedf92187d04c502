"""Batches of solids of more members than a launch grid's y dimension (65,535),
most of them too small for bricks (GPU)."""
import numpy as np
import pytest

from solvix_b200 import workloads

pytestmark = pytest.mark.gpu


def test_batch_of_more_members_than_a_grid_row(ctx):
    small = workloads.cantilever_c3d8(1, 1, 1, lx=0.1, ly=0.1, lz=0.1, seed=1)
    big = workloads.cantilever_c3d8(12, 4, 4, lx=1.2, ly=0.4, lz=0.4, seed=2)
    few, _ = ctx.solve_batch([small, big])
    flats = [small] * 65536
    flats[40000] = big
    out, stats = ctx.solve_batch(flats)
    assert stats["not_converged"] == 0
    # the brick member to the bit; the others run a CTA shape that is autotuned
    # for large classes, so to the bar of the plain batched solves
    np.testing.assert_array_equal(out[40000]["u"], few[1]["u"])
    assert out[40000]["iterations"] == few[1]["iterations"]
    for k in (0, 39999, 40001, 65535):
        err = np.linalg.norm(out[k]["u"] - few[0]["u"]) / np.linalg.norm(few[0]["u"])
        assert err <= 1e-10
