"""The chip-resident plane PCG (one cluster per model, K in registers)
against the oracle, at the sizes where its split changes: one CTA and two,
full and ragged thread counts, the largest model it takes and the first one
it does not, any node numbering, and meshes with a node of more than nine
neighbours, which take the general kernels (GPU).

The bar is the plain form's: u within 1e-10 of the oracle's (both stop at a
relative residual of 1e-10 on the same assembled K)."""
import numpy as np
import pytest

from oracle import oracle
from solvix_b200 import abi, workloads
from solvix_b200.marshal import FlatModel

pytestmark = pytest.mark.gpu

U_TOL = 1e-10


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def cantilever(nodes_x, nodes_y, seed=1):
    return workloads.cantilever_cps4(nodes_x - 1, nodes_y - 1, length=0.1 * (nodes_x - 1),
                                     height=0.1 * (nodes_y - 1), seed=seed)


def renumbered(flat, seed):
    """The same model with its nodes in a random order."""
    perm = np.random.default_rng(seed).permutation(flat.n_nodes)  # old -> new
    xyz = np.empty_like(flat.xyz)
    xyz[perm] = flat.xyz
    rows = perm[:, None] * 2 + np.arange(2)
    f = np.empty_like(flat.f)
    f[rows.ravel()] = flat.f
    return FlatModel(xyz=xyz, kind=flat.kind, conn_ptr=flat.conn_ptr, conn=perm[flat.conn],
                     youngs=flat.youngs, poisson=flat.poisson, thickness=flat.thickness, ndof=2,
                     fixed_row=rows.ravel()[flat.fixed_row], f=f), rows.ravel()


def disc(spokes, rings):
    """Triangles around a hub of `spokes` neighbours; the outer ring is held."""
    ang = 2 * np.pi * np.arange(spokes) / spokes
    xyz = [[0.0, 0.0, 0.0]]
    for r in range(1, rings + 1):
        xyz += [[r * np.cos(a), r * np.sin(a), 0.0] for a in ang]
    at = lambda r, s: 1 + (r - 1) * spokes + s % spokes  # noqa: E731
    tri = [[0, at(1, s), at(1, s + 1)] for s in range(spokes)]
    for r in range(1, rings):
        for s in range(spokes):
            tri += [[at(r, s), at(r + 1, s), at(r + 1, s + 1)],
                    [at(r, s), at(r + 1, s + 1), at(r, s + 1)]]
    n, m = len(xyz), len(tri)
    f = np.zeros(2 * n)
    f[0], f[2 * at(1, 1) + 1] = 300.0, -700.0
    held = np.array([at(rings, s) for s in range(spokes)])
    return FlatModel(xyz=np.array(xyz), kind=np.full(m, abi.SVX_CPS3, np.uint8),
                     conn_ptr=np.arange(m + 1) * 3, conn=np.array(tri).ravel(), youngs=2e9,
                     poisson=0.3, thickness=0.01, ndof=2,
                     fixed_row=np.stack([2 * held, 2 * held + 1], 1).ravel(), f=f)


@pytest.mark.parametrize("nodes", [(2, 2), (3, 11), (8, 8), (16, 16), (43, 6), (33, 31),
                                   (64, 32), (64, 64), (83, 50), (91, 90), (128, 64)])
def test_single_solves_at_the_edges_of_the_split(ctx, nodes):
    flat = cantilever(*nodes)
    sol, ref = ctx.solve_flat(flat), oracle.solve_flat(flat)
    assert rel(sol.u, ref.u) <= U_TOL and sol.final_residual <= 1e-10
    again = ctx.solve_flat(flat)
    assert np.array_equal(sol.u, again.u) and sol.iterations == again.iterations


@pytest.mark.parametrize("nodes", [(17, 9), (40, 20), (70, 64)])
def test_any_node_numbering(ctx, nodes):
    flat = cantilever(*nodes, seed=4)
    other, rows = renumbered(flat, 7)
    sol, ref = ctx.solve_flat(other), oracle.solve_flat(flat)
    assert rel(sol.u[rows], ref.u) <= U_TOL


def test_a_hub_of_many_neighbours_alone_and_in_a_batch(ctx):
    hub, plain = disc(12, 5), cantilever(32, 16)
    ref = oracle.solve_flat(hub)
    assert rel(ctx.solve_flat(hub).u, ref.u) <= U_TOL
    alone, _ = ctx.solve_batch([plain])
    out, st = ctx.solve_batch([plain, hub, plain])
    assert st["not_converged"] == 0
    assert rel(out[1]["u"], ref.u) <= U_TOL
    for k in (0, 2):
        assert np.array_equal(out[k]["u"], alone[0]["u"])


def test_batch_members_at_the_edges_of_the_split(ctx):
    sizes = [(2, 2), (8, 8), (5, 13), (32, 16), (27, 19), (64, 24), (64, 64), (70, 59), (91, 90),
             (128, 64)]
    flats = [cantilever(*s, seed=k) for k, s in enumerate(sizes)]
    out, st = ctx.solve_batch(flats)
    assert st["not_converged"] == 0
    for k, flat in enumerate(flats):
        ref = oracle.solve_flat(flat)
        assert rel(out[k]["u"], ref.u) <= U_TOL
        alone, _ = ctx.solve_batch([flat])
        assert np.array_equal(out[k]["u"], alone[0]["u"])


def test_budget_and_zero_load(ctx):
    flat = cantilever(64, 64)
    out, st = ctx.solve_batch([flat], max_iter=9)
    assert st["not_converged"] == 1 and out[0]["iterations"] == 9
    flat.f = np.zeros_like(flat.f)
    sol = ctx.solve_flat(flat)
    assert sol.iterations == 0 and not sol.u.any() and sol.final_residual == 0.0
