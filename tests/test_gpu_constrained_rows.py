"""Device memory of the constrained rows' copy: by the rows, not by the widest
node of the model (GPU).

One hub of 600 neighbours beside a plate whose 20,000 nodes are all held: at
the hub's width those 40,000 rows would take 580 MB, of their own 9.
"""
import numpy as np
import pytest
import torch

from oracle import oracle
from solvix_b200 import Context, abi, workloads
from solvix_b200.marshal import FlatModel

pytestmark = pytest.mark.gpu


def hub_and_plate(n=600):
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a), 0 * a], axis=1)
    xyz = np.vstack([np.zeros((1, 3)), ring, 2 * ring])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    t = np.vstack([np.stack([0 * i, 1 + i, 1 + j], axis=1),
                   np.stack([1 + i, 1 + n + i, 1 + n + j], axis=1),
                   np.stack([1 + i, 1 + n + j, 1 + j], axis=1)])
    p = workloads.cantilever_cps4(199, 99, length=19.9, height=9.9)
    shift = xyz.shape[0]
    f = np.zeros(2 * (shift + p.n_nodes))
    f[1] = 100.0
    outer = 1 + n + i
    fixed = np.concatenate([2 * outer, 2 * outer + 1, 2 * shift + np.arange(2 * p.n_nodes)])
    kind = np.concatenate([np.full(len(t), abi.SVX_CPS3, np.uint8), p.kind])
    nn = np.where(kind == abi.SVX_CPS3, 3, 4)
    return FlatModel(xyz=np.vstack([xyz, p.xyz + [5.0, 0.0, 0.0]]), kind=kind,
                     conn_ptr=np.concatenate([[0], np.cumsum(nn)]).astype(np.int64),
                     conn=np.concatenate([t.ravel(), p.conn + shift]).astype(np.int32),
                     youngs=1e9, poisson=0.3, thickness=0.1, ndof=2, fixed_row=fixed, f=f)


def test_rows_take_what_they_hold(ctx):
    flat = hub_and_plate()
    free0 = torch.cuda.mem_get_info()[0]
    with Context(0) as c:
        sol = c.solve_flat(flat)
        used = free0 - torch.cuda.mem_get_info()[0]
    assert used < 300e6
    ref = oracle.solve_flat(flat)
    assert np.linalg.norm(sol.u - ref.u) <= 1e-10 * np.linalg.norm(ref.u)
    scale = np.abs(ref.reaction_values).max()
    assert np.abs(sol.reaction_values - ref.reaction_values).max() <= 1e-8 * scale
