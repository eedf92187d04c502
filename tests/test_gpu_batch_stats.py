"""What a batch's statistics mean does not depend on the kernels its members
take (GPU)."""
import os

import pytest

from solvix_b200 import Context, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fresh():
    """A context of its own: the session's may have its CTA shape autotuned."""
    c = Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def on_k():
    old = {k: os.environ.get(k) for k in ("SVX_HEX", "SVX_RESIDENT")}
    os.environ.update({k: "0" for k in old})
    c = Context(0)
    for k, v in old.items():
        os.environ.pop(k) if v is None else os.environ.__setitem__(k, v)
    yield c
    c.close()


def hexes():
    # 288, 720, 3,075, 3,969 and 4,125 rows, the last one alone of cluster size
    sizes = [(5, 3, 3), (14, 3, 3), (40, 4, 4), (26, 6, 6), (54, 4, 4)]
    return [workloads.cantilever_c3d8(*s, lx=0.1 * s[0], ly=0.1 * s[1], lz=0.1 * s[2], seed=k)
            for k, s in enumerate(sizes)]


def plates():
    return [workloads.cantilever_cps4(nx, ny, length=0.1 * nx, height=0.1 * ny)
            for nx, ny in ((10, 4), (60, 12), (150, 40))]


@pytest.mark.parametrize("flats,clusters", [(hexes, 1), (plates, 0)])
def test_statistics_are_those_of_the_assembled_form(fresh, on_k, flats, clusters):
    flats = flats()
    assert sum(f.n_dof >= (4096 if f.ndof == 3 else 16384) for f in flats) == clusters
    _, new = fresh.solve_batch(flats)
    _, old = on_k.solve_batch(flats)
    for name in ("cluster_members", "threads_per_cta", "lanes_per_node", "total_dof"):
        assert new[name] == old[name], name
    assert new["cluster_members"] == clusters
