"""A wait between the CTAs of a cluster that runs out ends the solve with an
error, never with a hang (GPU).

The diagnostic form of the plane kernel drops one CTA's sums, or lets a third
of its threads take the wait to have run out although the sums came: the CTA
must leave as one, the others' waits run out in turn, and the context solves
on.  Nothing here faults the GPU, and every wait of the kernel is bounded.
"""
import ctypes as C
import time

import numpy as np
import pytest

from solvix_b200 import abi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(40, 7), (100, 10), (200, 20)])  # 3, 9 and 16 CTAs
@pytest.mark.parametrize("fault", [0, 1, 2, 3])
def test_wait_that_runs_out_is_an_error(ctx, size, fault):
    lib = abi.load()
    flat = workloads.cantilever_cps4(*size, length=0.1 * size[0], height=0.1 * size[1])
    op = ctx.assemble(flat)
    before = op.solve()
    err = abi.SvxError()
    t = time.perf_counter()
    st = lib.svx_diag_resident_stall(op.handle, fault, 2000, C.byref(err))
    assert time.perf_counter() - t < 1.0
    assert st == abi.SVX_CUDA_ERROR and b"ran out" in err.message
    after = op.solve()
    np.testing.assert_array_equal(after[0], before[0])
    assert after[1] == before[1]
    op.free()


def test_stall_diagnostic_rejects_what_it_cannot_run(ctx):
    lib = abi.load()
    err = abi.SvxError()
    one = ctx.assemble(workloads.cantilever_cps4(10, 4, length=1.0, height=0.4))
    assert lib.svx_diag_resident_stall(one.handle, 0, 1000, C.byref(err)) == abi.SVX_BAD_ARGUMENT
    two = ctx.assemble(workloads.cantilever_cps4(100, 10, length=10.0))
    for fault, wait in ((-1, 1000), (4, 1000), (0, 0), (0, 1 << 30)):
        assert lib.svx_diag_resident_stall(two.handle, fault, wait,
                                           C.byref(err)) == abi.SVX_BAD_ARGUMENT
    one.free()
    two.free()
