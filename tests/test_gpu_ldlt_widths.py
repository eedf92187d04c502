"""The direct path at the bandwidths where its substitutions change form: the
one-block form takes one tile a warp up to a half-bandwidth of 16 tiles of 32
(each tile alone, the last warp's, one more), the factorization steps at the
ends of the band, and systems of one, two and three block rows.

Bars as for the other direct solves: u within 1e-8 relative of the oracle's,
the condition estimate within 1e-6, the residual within 1e-8."""
import numpy as np
import pytest

from oracle import oracle
from solvix_b200 import solve_with_method
from solvix_b200.model import Method
from svx_cases import hex_cantilever
from test_ldlt_host import product_rcm
from test_oracle_ldlt import modified_system

pytestmark = pytest.mark.gpu

# dims: half-bandwidth in tiles in the reference's ordering
WIDTHS = {(1, 1, 1): 1, (2, 1, 1): 1, (5, 1, 1): 1, (9, 2, 1): 2, (9, 2, 2): 3, (14, 4, 4): 7,
          (14, 7, 6): 15, (20, 15, 4): 16, (22, 16, 4): 17, (14, 7, 7): 18}


@pytest.mark.parametrize("dims", sorted(WIDTHS))
def test_direct_solves_by_bandwidth(ctx, dims):
    m = hex_cantilever(*dims)
    k, f, _ = modified_system(m)
    assert -(-product_rcm(k)[1] // 32) == WIDTHS[dims]
    ref = oracle.ldlt(k, f)
    sol = solve_with_method(m, Method.Ldlt, ctx=ctx)
    assert sol.final_residual <= 1e-8
    assert np.linalg.norm(sol.u - ref.u) <= 1e-8 * np.linalg.norm(ref.u)
    assert abs(sol.cond_estimate - ref.cond) <= 1e-6 * ref.cond
