"""A host that refuses the page-locked staging buffer: single solves copy from
and to the caller's arrays (GPU)."""
import os

import numpy as np
import pytest

from solvix_b200 import Context, workloads
from solvix_b200.model import DeviceError, NotConverged

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bare():
    old = os.environ.get("SVX_STAGING_MAX")
    os.environ["SVX_STAGING_MAX"] = "0"
    c = Context(0)
    os.environ.pop("SVX_STAGING_MAX") if old is None else \
        os.environ.__setitem__("SVX_STAGING_MAX", old)
    yield c
    c.close()


@pytest.mark.parametrize("flat", [
    workloads.cantilever_cps4(30, 6, length=3.0, height=0.6),
    workloads.cantilever_c3d8(12, 3, 3, lx=1.2, ly=0.3, lz=0.3, seed=2)])
def test_single_solves_need_no_page_locked_memory(ctx, bare, flat):
    a, b = ctx.solve_flat(flat), bare.solve_flat(flat)
    for name in ("u", "von_mises", "nodal_von_mises", "reaction_values", "displacements"):
        np.testing.assert_array_equal(getattr(a, name), getattr(b, name))
    with pytest.raises(NotConverged):
        bare.solve_flat(flat, max_iter=3)
    op = bare.assemble(flat)
    op.solve()
    np.testing.assert_array_equal(op.stress()[0], a.von_mises)
    op.free()


def test_batches_still_report_it(bare):
    flat = workloads.cantilever_cps4(30, 6, length=3.0, height=0.6)
    with pytest.raises(DeviceError):
        bare.solve_batch([flat])
