"""The members of a batch that stay on the assembled K run beside those on
clusters, not after them (GPU).

Five one-CTA members and one 16-CTA member leave most of the device idle, so
together they take the time of the longer kind; run one after the other they
would take the sum.  The line is drawn half way.
"""
import numpy as np
import pytest

from solvix_b200 import workloads
from solvix_b200.marshal import FlatModel

pytestmark = pytest.mark.gpu


def with_orphan(f):
    """The model and a node that no element uses: such a member stays on K."""
    n = f.n_nodes
    return FlatModel(xyz=np.vstack([f.xyz, [9.0, 9.0, 9.0]]), kind=f.kind, conn_ptr=f.conn_ptr,
                     conn=f.conn, youngs=f.youngs, poisson=f.poisson, thickness=f.thickness,
                     ndof=3, fixed_row=np.concatenate([f.fixed_row, 3 * n + np.arange(3)]),
                     f=np.concatenate([f.f, np.zeros(3)]))


def test_one_cta_members_run_beside_clusters(ctx):
    on_k = [with_orphan(workloads.cantilever_c3d8(40, 4, 4, lx=4.0, ly=0.4, lz=0.4, seed=k))
            for k in range(5)]
    cluster = [workloads.cantilever_c3d8(110, 16, 16, lx=11.0, ly=1.6, lz=1.6, seed=9)]

    def ms(flats):
        runs = [ctx.solve_batch(flats)[1] for _ in range(4)]
        assert all(r["not_converged"] == 0 for r in runs)
        return min(r["ms_solve"] for r in runs[1:])

    a, b, both = ms(on_k), ms(cluster), ms(on_k + cluster)
    assert min(a, b) > 3.0, (a, b)  # long enough to tell
    assert both < a + b - 0.5 * min(a, b), (a, b, both)
