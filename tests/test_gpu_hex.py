"""The element-by-element operator of C3D8 models (GPU): the graph form, the
whole-device form on bricks and the batch's clusters, against the oracle's
solves on the assembled K, at the sizes where the split changes: one brick
and many, chunks that are full and nearly empty, members of one to sixteen
CTAs, any node numbering, nodes that many bricks share, and members with a
node no element uses, which keep the assembled K.

The bar is the plain form's 1e-10 on u: the operator equals K up to rounding,
which these models (not slender) amplify to some 1e-12."""
import numpy as np
import pytest

from oracle import oracle
from solvix_b200 import Context, abi, workloads
from solvix_b200.marshal import FlatModel

pytestmark = pytest.mark.gpu

U_TOL = 1e-10


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def block(nx, ny, nz, seed=1, hetero=None):
    return workloads.cantilever_c3d8(nx, ny, nz, lx=0.1 * nx, ly=0.1 * ny, lz=0.1 * nz,
                                     seed=seed, hetero_E=hetero)


def renumbered(flat, seed):
    perm = np.random.default_rng(seed).permutation(flat.n_nodes)
    xyz = np.empty_like(flat.xyz)
    xyz[perm] = flat.xyz
    rows = (perm[:, None] * 3 + np.arange(3)).ravel()
    f = np.empty_like(flat.f)
    f[rows] = flat.f
    return FlatModel(xyz=xyz, kind=flat.kind, conn_ptr=flat.conn_ptr, conn=perm[flat.conn],
                     youngs=flat.youngs, poisson=flat.poisson, thickness=1.0, ndof=3,
                     fixed_row=rows[flat.fixed_row], f=f), rows


def with_orphan(flat):
    n = flat.n_nodes
    return FlatModel(xyz=np.vstack([flat.xyz, [[9.0, 9.0, 9.0]]]), kind=flat.kind,
                     conn_ptr=flat.conn_ptr, conn=flat.conn, youngs=flat.youngs,
                     poisson=flat.poisson, thickness=1.0, ndof=3,
                     fixed_row=np.concatenate([flat.fixed_row, 3 * n + np.arange(3)]),
                     f=np.concatenate([flat.f, np.zeros(3)]))


@pytest.fixture(scope="module")
def forms():
    """Contexts whose C3D8 solves of any size take the bricks, and the graph
    form."""
    mp = pytest.MonkeyPatch()
    mp.setenv("SVX_HEX_MIN_NODES", "0")
    bricks = Context(0)
    mp.setenv("SVX_BRICK_MAX_ELEMS", "1")
    graph = Context(0)
    mp.undo()
    yield {"bricks": bricks, "graph": graph}
    bricks.close()
    graph.close()


SIZES = [(2, 1, 1), (8, 4, 4), (16, 4, 2), (43, 3, 1), (33, 8, 8), (24, 16, 5), (12, 12, 12)]


@pytest.mark.parametrize("form", ["bricks", "graph"])
@pytest.mark.parametrize("size", SIZES)
def test_forms_match_the_oracle(forms, form, size):
    flat = block(*size, hetero=(9.5, 10.5) if size[0] == 24 else None)
    sol, ref = forms[form].solve_flat(flat), oracle.solve_flat(flat)
    assert rel(sol.u, ref.u) <= U_TOL and sol.final_residual <= 1e-10
    again = forms[form].solve_flat(flat)
    assert np.array_equal(sol.u, again.u) and sol.iterations == again.iterations


@pytest.mark.parametrize("form", ["bricks", "graph"])
def test_numbering_orphans_and_budget(forms, form):
    flat = block(20, 5, 4, seed=3)
    ref = oracle.solve_flat(flat)
    other, rows = renumbered(flat, 5)
    assert rel(forms[form].solve_flat(other).u[rows], ref.u) <= U_TOL
    assert rel(forms[form].solve_flat(with_orphan(flat)).u[: flat.n_dof], ref.u) <= U_TOL
    mixed = forms[form].solve_flat(flat, precision=abi.SVX_MIXED)
    assert rel(mixed.u, ref.u) <= 1e-8 and mixed.final_residual <= 1e-10
    from solvix_b200.model import NotConverged
    with pytest.raises(NotConverged) as e:
        forms[form].solve_flat(flat, max_iter=11)
    assert e.value.iterations == 11


def test_default_context_takes_the_forms_by_size(ctx):
    for size in ((60, 16, 16), (184, 16, 16)):
        flat = block(*size)
        assert rel(ctx.solve_flat(flat).u, oracle.solve_flat(flat).u) <= U_TOL


def test_batch_members_of_one_to_sixteen_ctas(ctx):
    """Members of every cluster size; each the same alone and in the mix."""
    sizes = [(10, 3, 3), (30, 7, 7), (32, 7, 7), (25, 16, 4), (30, 10, 10), (41, 14, 14),
             (64, 16, 16)]
    flats = [block(*s, seed=k) for k, s in enumerate(sizes)]
    flats.append(with_orphan(flats[3]))
    out, st = ctx.solve_batch(flats)
    assert st["not_converged"] == 0
    for k, flat in enumerate(flats):
        ref = oracle.solve_flat(flat)
        assert rel(out[k]["u"], ref.u) <= U_TOL, k
    for k in (2, 4, 6):
        alone, _ = ctx.solve_batch([flats[k]])
        assert np.array_equal(alone[0]["u"], out[k]["u"])
        assert alone[0]["iterations"] == out[k]["iterations"]


@pytest.mark.parametrize("size", [(4, 3, 3), (5, 3, 3), (6, 3, 3), (20, 4, 4), (33, 4, 4)])
def test_small_batch_members(ctx, size):
    """Members about the batch's threshold of 96 nodes (80, 96, 112) and of one
    and two CTAs (320 and 528 elements), beside a model above it and one that
    keeps K."""
    flats = [block(*size, seed=7), block(12, 5, 5, seed=8), with_orphan(block(*size, seed=9))]
    out, st = ctx.solve_batch(flats)
    assert st["not_converged"] == 0
    for k, flat in enumerate(flats):
        assert rel(out[k]["u"], oracle.solve_flat(flat).u) <= U_TOL, k
    alone, _ = ctx.solve_batch(flats[:1])
    assert np.array_equal(alone[0]["u"], out[0]["u"])
    assert alone[0]["iterations"] == out[0]["iterations"]


@pytest.mark.parametrize("size", [(3, 1, 1), (20, 5, 4), (48, 9, 8)])
def test_defect_correction_below_the_graph_threshold(ctx, size):
    """The FP32 inner solves on the shared-memory kernel, of one node a block
    to several (and the plane form's two barriers)."""
    flat = block(*size, hetero=(9.0, 11.0))
    sol, ref = ctx.solve_flat(flat, precision=abi.SVX_MIXED_DEFECT), oracle.solve_flat(flat)
    assert sol.final_residual <= 1e-10 and 0 < sol.fp32_iterations <= sol.iterations
    assert rel(sol.u, ref.u) <= 1e-8
    plane = workloads.cantilever_cps4(10 * size[1], 4 * size[2], length=size[1],
                                      height=0.4 * size[2])
    sol = ctx.solve_flat(plane, precision=abi.SVX_MIXED_DEFECT)
    assert rel(sol.u, oracle.solve_flat(plane).u) <= 1e-8
