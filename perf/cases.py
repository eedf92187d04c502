"""The work whose time this framework is judged by, through its public entry
points: single solves from host arrays (plane and solid, FP64 and the two
mixed forms, iterative and direct), a solve on an operator kept on the
device, batched solves, served requests and steady conduction.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes the inputs of a case from a seed (and what a program
keeps between calls: the context, the assembled operator, the server),
``run`` is one call, ``work`` the bytes and operations that call cannot do
without and ``exact`` its results in 64-bit torch arithmetic.

Results are the solved fields.  The number of CG iterations is left out: it
is the length of the path to a solution, not part of it, and moves with the
order in which a dot product is summed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from solvix_b200 import abi, workloads
from solvix_b200.core import default_context
from solvix_b200.marshal import ThermalModel
from solvix_b200.serve import Server

CPS3, CPS4, C3D8 = abi.SVX_CPS3, abi.SVX_CPS4, abi.SVX_C3D8
PRECISION = {"fp64": abi.SVX_FP64, "mixed": abi.SVX_MIXED, "defect": abi.SVX_MIXED_DEFECT}
# elements of length per element of height at most: a longer bare strip
# amplifies the rounding of its 64-bit stiffness matrix into digits that a
# comparison of two correct solvers would see
SLENDER = 12
METHOD = {"pcg": abi.SVX_METHOD_PCG, "ldlt": abi.SVX_METHOD_LDLT}


def listed():
    return [
        # the smallest plate of the 2D mix, solved from host arrays to host
        # fields: a request-sized call, where latency and launches count
        {"name": "plate 10x4", "what": "plane", "kind": "cps4", "nx": 10, "ny": 4},
        # the jittered 200 x 20 plane-stress cantilever (8,442 DOF): the
        # ordinary 2D analysis and the smallest published configuration
        {"name": "cantilever 200x20", "what": "cantilever", "nx": 200, "ny": 20},
        # a triangulated plate of odd sizes near the top of the 2D mix
        {"name": "plate 133x37 cps3", "what": "plane", "kind": "cps3", "nx": 133, "ny": 37},
        # a 256-plate share of the 4,096-plate mix, one batched call: uneven
        # sizes (nx to 160, ny 4 to 40), CPS3 and CPS4 members side by side
        {"name": "batch of 256 plates", "what": "batch", "of": "plates", "count": 256,
         "mix": 1, "precision": "fp64"},
        # a batch of the serving mix's 3D cantilevers
        {"name": "batch of 40 hex", "what": "batch", "of": "hexes", "count": 40,
         "mix": 2, "precision": "fp64"},
        # requests of the serving mix (70 % plates, 30 % hex cantilevers)
        # submitted at once to a running server and polled until done
        {"name": "serve 96 requests", "what": "serve", "count": 96, "mix": 3,
         "precision": "fp64"},
        # the direct path on the mesh of the reference's own LDLt timing
        {"name": "hex 40x4x4 direct", "what": "solid", "nx": 40, "ny": 4, "nz": 4,
         "hetero": False, "precision": "fp64", "method": "ldlt"},
        # the 160 x 16 x 16 solid cantilever (139,587 DOF), K inside L2:
        # the ordinary 3D analysis, host arrays to host fields
        {"name": "hex 160x16x16", "what": "solid", "nx": 160, "ny": 16, "nz": 16,
         "hetero": False, "precision": "fp64", "method": "pcg"},
        # the relaxed mixed form on a heterogeneous solid
        {"name": "hex 160x16x16 mixed", "what": "solid", "nx": 160, "ny": 16, "nz": 16,
         "hetero": True, "precision": "mixed", "method": "pcg"},
        # the FP32 inner / FP64 outer form on a smaller heterogeneous solid
        {"name": "hex 80x8x8 defect", "what": "solid", "nx": 80, "ny": 8, "nz": 8,
         "hetero": True, "precision": "defect", "method": "pcg"},
        # a large heterogeneous solid (1.05M DOF, K 0.65 GB, beyond L2) on
        # an operator assembled once and kept, as a program that solves for
        # load after load keeps it
        {"name": "hex 320x32x32 kept", "what": "kept", "nx": 320, "ny": 32, "nz": 32},
        # steady conduction in a solid block, host model to temperatures
        {"name": "conduction 240x24x24", "what": "conduction", "nx": 240, "ny": 24, "nz": 24},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case; element counts stay within the listed ones'."""
    what = rng.choice(["plane", "plane", "cantilever", "batch", "batch", "serve", "solid",
                       "solid", "solid", "direct", "kept", "conduction"])
    if what == "plane":
        ny = _log(rng, 4, 40)
        return {"what": what, "kind": rng.choice(["cps3", "cps4"]),
                "nx": _log(rng, 10, min(160, SLENDER * ny)), "ny": ny}
    if what == "cantilever":
        ny = _log(rng, 4, 40)
        return {"what": what, "nx": _log(rng, 20, min(300, SLENDER * ny)), "ny": ny}
    if what == "batch":
        of = rng.choice(["plates", "plates", "hexes"])
        return {"what": what, "of": of,
                "count": _log(rng, 4, 256) if of == "plates" else _log(rng, 2, 40),
                "mix": rng.randrange(1 << 20), "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if what == "serve":
        return {"what": what, "count": _log(rng, 8, 96), "mix": rng.randrange(1 << 20),
                "precision": "fp64"}
    if what == "solid":
        precision = rng.choice(["fp64", "fp64", "mixed", "defect"])
        top = 80 if precision == "defect" else 160
        nx = _log(rng, 8, top)
        lim = max(2, min(16, nx // 4))
        return {"what": what, "nx": nx, "ny": _log(rng, 2, lim), "nz": _log(rng, 2, lim),
                "hetero": rng.random() < 0.5, "precision": precision, "method": "pcg"}
    if what == "direct":
        nx = _log(rng, 8, 48)
        return {"what": "solid", "nx": nx, "ny": rng.randint(2, 5), "nz": rng.randint(2, 5),
                "hetero": False, "precision": "fp64", "method": "ldlt"}
    if what == "kept":
        return {"what": what, "nx": _log(rng, 120, 300), "ny": rng.randint(17, 32),
                "nz": rng.randint(17, 32)}
    return {"what": what, "nx": _log(rng, 12, 240), "ny": _log(rng, 4, 24),
            "nz": _log(rng, 4, 24)}


# ------------------------------------------------------------------ inputs
def _seed(case, seed):
    """The generator of one case's inputs: other cases and seeds, other inputs."""
    key = [seed & 0x7fffffff] + [ord(c) for k in sorted(case) if k != "name"
                                 for c in "%s=%s;" % (k, case[k])]
    return np.random.Generator(np.random.PCG64(np.random.SeedSequence(key)))


def _plate(rng, kind, nx, ny):
    """A plate of the 2D mix of the given element kind and size."""
    flat = workloads.plate(rng, nx, ny)
    while flat.kind[0] != kind:
        flat = workloads.plate(rng, nx, ny)
    return flat


def _hex_member(rng, nx, nyz):
    """A 3D cantilever of the serving mix of the given size."""
    return workloads.cantilever_c3d8(nx, nyz, nyz, lx=nx / nyz * 0.1, ly=0.1, lz=0.1,
                                     jitter=0.0, E=70e9, nu=0.33,
                                     total_load=-rng.uniform(1e3, 1e4))


def _members(case, rng):
    """The members of a batch or a served mix: element kinds and sizes follow
    the case's "mix" number, materials and loads the seed."""
    sizes = np.random.Generator(np.random.PCG64(case["mix"]))
    share = {"plates": 1.0, "hexes": 0.0, "requests": 0.7}[case.get("of", "requests")]
    out = []
    for _ in range(case["count"]):
        if sizes.random() < share:
            kind = CPS3 if sizes.random() < 0.5 else CPS4
            ny = int(sizes.integers(4, 41))
            out.append(_plate(rng, kind, int(sizes.integers(10, min(160, SLENDER * ny) + 1)), ny))
        else:
            nyz = int(sizes.integers(4, 17))
            nx = int(sizes.integers(20, min(120, SLENDER * nyz) + 1))
            out.append(_hex_member(rng, nx, nyz))
    return out


def _conduction(case, rng):
    """A solid block with random interior offsets, hot and cold end faces and
    a volumetric source."""
    flat = workloads.cantilever_c3d8(case["nx"], case["ny"], case["nz"], jitter=0.1,
                                     seed=int(rng.integers(1 << 31)))
    per = case["nx"] + 1
    i = np.arange(flat.n_nodes) % per
    cold, hot = np.flatnonzero(i == 0), np.flatnonzero(i == case["nx"])
    return ThermalModel(flat.xyz, flat.kind, flat.conn_ptr, flat.conn,
                        float(rng.uniform(15.0, 60.0)), source=float(rng.uniform(5e4, 2e5)),
                        temp_node=np.concatenate([cold, hot]),
                        temp_value=np.concatenate([np.full(cold.size, 20.0),
                                                   np.full(hot.size, rng.uniform(60, 90))]))


def _models(case, seed):
    """The flat models of a case (a list), or its conduction model."""
    rng = _seed(case, seed)
    what = case["what"]
    if what == "plane":
        kind = CPS3 if case["kind"] == "cps3" else CPS4
        return [_plate(rng, kind, case["nx"], case["ny"])]
    if what == "cantilever":
        return [workloads.cantilever_cps4(case["nx"], case["ny"], length=0.05 * case["nx"],
                                          height=0.05 * case["ny"],
                                          load=-float(rng.uniform(500, 2000)),
                                          seed=int(rng.integers(1 << 31)))]
    if what in ("solid", "kept"):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        h = 0.0125
        het = what == "kept" or case["hetero"]
        return [workloads.cantilever_c3d8(nx, ny, nz, lx=h * nx, ly=h * ny, lz=h * nz,
                                          total_load=-float(rng.uniform(2e3, 8e3)),
                                          hetero_E=(9.0, 11.0) if het else None,
                                          nu=0.3 if het else 0.33,
                                          seed=int(rng.integers(1 << 31)))]
    if what in ("batch", "serve"):
        return _members(case, rng)
    return _conduction(case, rng)


def prepare(case, seed):
    ctx = default_context()
    models = _models(case, seed)
    state = {"case": case, "ctx": ctx, "models": models}
    if case["what"] == "kept":
        state["op"] = ctx.assemble(models[0])
    elif case["what"] == "serve":
        state["server"] = Server(hbm_budget_bytes=8 << 30,
                                 precision=PRECISION[case["precision"]])
    return state


def run(state):
    case, ctx, models = state["case"], state["ctx"], state["models"]
    what = case["what"]
    if what == "conduction":
        return ctx.solve_thermal(models)[0]
    if what == "kept":
        u, _, _, cond = state["op"].solve()
        return {"u": u, "cond": cond}
    if what == "batch":
        out, _ = ctx.solve_batch(models, precision=PRECISION[case["precision"]])
        return {"u": np.concatenate([o["u"] for o in out]),
                "von_mises": np.concatenate([o["von_mises"] for o in out])}
    if what == "serve":
        server = state["server"]
        for k, flat in enumerate(models):
            status, message = server.submit(flat, k)
            if status != abi.SVX_OK:
                raise RuntimeError(message)
        got = {}
        while len(got) < len(models):
            r = server.poll()
            got[r["tag"]] = r
        return {"u": np.concatenate([got[k]["u"] for k in range(len(models))]),
                "von_mises": np.concatenate([got[k]["von_mises"] for k in range(len(models))])}
    sol = ctx.solve_flat(models[0], precision=PRECISION[case.get("precision", "fp64")],
                         method=METHOD[case.get("method", "pcg")])
    return {"u": sol.u, "displacements": sol.displacements, "von_mises": sol.von_mises,
            "nodal_von_mises": sol.nodal_von_mises, "reactions": sol.reaction_values}


# -------------------------------------------------------------------- work
def _counts(what, nx, ny, nz=0, tri=False):
    """(nodes, elements, element nodes, dofs per node) of a structured mesh."""
    if what in ("plane", "cantilever"):
        return (nx + 1) * (ny + 1), nx * ny * (2 if tri else 1), 3 if tri else 4, 2
    nd = 1 if what == "conduction" else 3
    return (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz, 8, nd


def _model_work(nodes, elems, nn, nd):
    """The model in (coordinates, loads, connectivity, material), the fields
    out, the integration of every element matrix once and the operator
    applied once per element along the longest way a load travels (a Krylov
    solver cannot reach a far node in fewer applications); a mesh of N
    elements in d dimensions is at least N^(1/d) of them across."""
    across = elems ** (0.5 if nd == 2 else 1.0 / 3.0)
    n = nn * nd
    s = {1: 3, 2: 3, 3: 6}[nd]
    points = {3: 1, 4: 4, 8: 8}[nn]
    flops = elems * (points * n * (n + 1) * s + 2.0 * n * n * across)
    return {"bytes": 24.0 * nodes + 16.0 * nd * nodes + elems * (4.0 * nn + 33.0),
            "flops": flops}


def work(case):
    what = case["what"]
    if what in ("batch", "serve"):
        # the mean member of the mixes: plates of 85 x 22, hexes of 70 x 10 x 10
        plate = _model_work(*_counts("plane", 85, 22))
        block = _model_work(*_counts("solid", 70, 10, 10))
        share = {"plates": 1.0, "hexes": 0.0}[case["of"]] if what == "batch" else 0.7
        return {k: case["count"] * (share * plate[k] + (1 - share) * block[k]) for k in plate}
    return _model_work(*_counts(what, case["nx"], case["ny"], case.get("nz", 0),
                                case.get("kind") == "cps3"))


# ------------------------------------------------------------------- exact
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


_CORNERS = {
    CPS4: [(-1, -1), (1, -1), (1, 1), (-1, 1)],
    C3D8: [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1),
           (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)],
}


def _grad(kind, x, point):
    """Physical shape-function gradients [E, nn, dim] and the Jacobian (or
    area) weight [E] at a natural point.  For solids the inverse Jacobian is
    the published method's: the cofactors of odd index sum change sign."""
    if kind == CPS3:
        a, b, c = x[:, 0], x[:, 1], x[:, 2]
        gx = torch.stack([b[:, 1] - c[:, 1], c[:, 1] - a[:, 1], a[:, 1] - b[:, 1]], 1)
        gy = torch.stack([c[:, 0] - b[:, 0], a[:, 0] - c[:, 0], b[:, 0] - a[:, 0]], 1)
        two = gx[:, 0] * gy[:, 1] - gx[:, 1] * gy[:, 0]
        return torch.stack([gx, gy], 2) / two[:, None, None], two.abs() / 2.0
    corners = torch.tensor(_CORNERS[kind], dtype=torch.float64, device=x.device)
    dim = corners.shape[1]
    terms = 1.0 + corners * torch.tensor(point, dtype=torch.float64, device=x.device)
    dn = torch.stack([corners[:, a] * torch.stack(
        [terms[:, b] for b in range(dim) if b != a], 0).prod(0) for a in range(dim)], 0)
    dn = dn / 2.0 ** dim                                   # [dim, nn]
    jac = torch.einsum("an,enb->eab", dn, x[:, :, :dim])
    det = torch.linalg.det(jac)
    if dim == 3 and kind == C3D8:
        rows = []
        for r in range(3):
            for c in range(3):
                i, j = (r + 1) % 3, (r + 2) % 3
                k, m = (c + 1) % 3, (c + 2) % 3
                cof = jac[:, i, k] * jac[:, j, m] - jac[:, i, m] * jac[:, j, k]
                rows.append(cof if (r + c) % 2 == 0 else -cof)
        inv = torch.stack(rows, 1).reshape(-1, 3, 3).transpose(1, 2) / det[:, None, None]
    else:
        inv = torch.linalg.inv(jac)
    return torch.einsum("eba,an->enb", inv, dn), det


def _points(kind):
    if kind == CPS3:
        return [(0.0, 0.0)]
    g, dim = 1.0 / math.sqrt(3.0), 2 if kind == CPS4 else 3
    return [tuple((g if (p >> (dim - 1 - a)) & 1 else -g) for a in range(dim))
            for p in range(2 ** dim)]


def _bmat(grad):
    """Strain-displacement matrices [E, S, nn * dim] of gradients."""
    e, nn, dim = grad.shape
    if dim == 2:
        b = torch.zeros(e, 3, nn, 2, dtype=grad.dtype, device=grad.device)
        b[:, 0, :, 0], b[:, 1, :, 1] = grad[..., 0], grad[..., 1]
        b[:, 2, :, 0], b[:, 2, :, 1] = grad[..., 1], grad[..., 0]
    else:
        b = torch.zeros(e, 6, nn, 3, dtype=grad.dtype, device=grad.device)
        for a in range(3):
            b[:, a, :, a] = grad[..., a]
        b[:, 3, :, 0], b[:, 3, :, 1] = grad[..., 1], grad[..., 0]
        b[:, 4, :, 1], b[:, 4, :, 2] = grad[..., 2], grad[..., 1]
        b[:, 5, :, 0], b[:, 5, :, 2] = grad[..., 2], grad[..., 0]
    return b.reshape(e, b.shape[1], -1)


def _dmat(kind, E, nu):
    """Elasticity matrices [E, S, S] (plane stress or solid)."""
    d = torch.zeros(E.shape[0], 3 if kind != C3D8 else 6, 3 if kind != C3D8 else 6,
                    dtype=E.dtype, device=E.device)
    if kind != C3D8:
        c = E / (1.0 - nu * nu)
        d[:, 0, 0] = d[:, 1, 1] = c
        d[:, 0, 1] = d[:, 1, 0] = nu * c
        d[:, 2, 2] = c * (1.0 - nu) / 2.0
        return d
    lam, mu = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), E / (2.0 * (1.0 + nu))
    d[:, :3, :3] = lam[:, None, None]
    for a in range(3):
        d[:, a, a] += 2.0 * mu
        d[:, 3 + a, 3 + a] = mu
    return d


def _cg(groups, f, free, member, count):
    """K u = f on the free rows by Jacobi-CG with one scalar set per member,
    restarted from the true residual until it is at rounding level.  groups:
    (dof indices [E, N], element matrices [E, N, N])."""
    def apply(x):
        y = torch.zeros_like(x)
        for dofs, ke in groups:
            y.index_add_(0, dofs.reshape(-1),
                         torch.bmm(ke, x[dofs].unsqueeze(2)).reshape(-1))
        return y * free

    def dots(a, b):
        if count == 1:
            return torch.dot(a, b).reshape(1)
        return torch.zeros(count, dtype=a.dtype, device=a.device).index_add_(0, member, a * b)

    diag = torch.zeros_like(f)
    for dofs, ke in groups:
        diag.index_add_(0, dofs.reshape(-1), ke.diagonal(dim1=1, dim2=2).reshape(-1))
    inv = torch.where(free.bool() & (diag != 0), 1.0 / diag, torch.zeros_like(diag))
    b = f * free
    norm = dots(b, b).sqrt().clamp_min(1e-300)
    u = torch.zeros_like(b)
    for outer in range(3):
        r = b - apply(u)
        if bool(((dots(r, r).sqrt() / norm) < 1e-14).all()):
            break
        start = dots(r, r).sqrt().clamp_min(1e-300)
        p = torch.zeros_like(r)
        e = torch.zeros_like(r)
        rz = torch.ones_like(norm)
        goal = 1e-14 if outer == 0 else 1e-6
        beta = torch.zeros_like(rz)
        for it in range(60000):
            z = r * inv
            rz_new = dots(r, z)
            beta = torch.where(rz > 0, rz_new / rz, torch.zeros_like(rz)) if it else beta
            p = z + (beta if count == 1 else beta[member]) * p
            rz = rz_new
            q = apply(p)
            pq = dots(p, q)
            alpha = torch.where(pq > 0, rz / pq, torch.zeros_like(pq))
            am = alpha if count == 1 else alpha[member]
            e += am * p
            r = r - am * q
            if it % 50 == 49 and bool(((dots(r, r).sqrt() / start) <= goal).all()):
                break
        u = u + e
    return u


def _von_mises(s):
    if s.shape[1] == 3:
        return torch.sqrt(0.5 * ((s[:, 0] - s[:, 1]) ** 2 + s[:, 1] ** 2 + s[:, 0] ** 2)
                          + 3.0 * s[:, 2] ** 2)
    return torch.sqrt(0.5 * ((s[:, 0] - s[:, 1]) ** 2 + (s[:, 1] - s[:, 2]) ** 2
                             + (s[:, 2] - s[:, 0]) ** 2) + 3.0 * (s[:, 3:] ** 2).sum(1))


class _System:
    """Members of one ndof as one block-diagonal 64-bit system."""

    def __init__(self, flats):
        dev = _device()
        nd = flats[0].ndof
        self.nd, self.parts, self.groups = nd, [], []
        nodes = np.cumsum([0] + [f.n_nodes for f in flats])
        elems = np.cumsum([0] + [f.n_elem for f in flats])
        self.n_nodes, self.n_elem = int(nodes[-1]), int(elems[-1])
        t = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a),  # noqa: E731
                                                        dtype=dt, device=dev)
        xyz = t(np.concatenate([f.xyz for f in flats]))
        kinds = np.concatenate([f.kind for f in flats])
        E = t(np.concatenate([f.youngs for f in flats]))
        nu = t(np.concatenate([f.poisson for f in flats]))
        th = t(np.concatenate([np.full(f.n_elem, f.thickness) for f in flats]))
        first = np.concatenate([f.conn_ptr[:-1] + c for f, c in zip(
            flats, np.cumsum([0] + [f.conn.size for f in flats]))])
        conn = np.concatenate([f.conn.astype(np.int64) + o for f, o in zip(flats, nodes)])
        for kind, nn in ((CPS3, 3), (CPS4, 4), (C3D8, 8)):
            at = np.flatnonzero(kinds == kind)
            if not at.size:
                continue
            c = t(conn[first[at][:, None] + np.arange(nn)], torch.int64)
            ids = t(at, torch.int64)
            x, d = xyz[c], _dmat(kind, E[ids], nu[ids])
            ke = 0.0
            for p in _points(kind):
                grad, w = _grad(kind, x, p)
                b = _bmat(grad)
                w = w * th[ids] if nd == 2 else w
                ke = ke + torch.bmm(b.transpose(1, 2), torch.bmm(d, b)) * w[:, None, None]
            dofs = (c[:, :, None] * nd + torch.arange(nd, device=dev)).reshape(c.shape[0], -1)
            self.groups.append((dofs, ke))
            self.parts.append((kind, ids, c, dofs, x, d))
        self.f = t(np.concatenate([f.f for f in flats]))
        fixed = t(np.concatenate([f.fixed_row + o * nd for f, o in zip(flats, nodes)]),
                  torch.int64)
        self.fixed = fixed
        free = torch.ones_like(self.f)
        free[fixed] = 0.0
        member = t(np.repeat(np.arange(len(flats)), np.diff(nodes) * nd), torch.int64)
        self.u = _cg(self.groups, self.f, free, member, len(flats))

    def centroid(self):
        vm = torch.zeros(self.n_elem, dtype=torch.float64, device=self.u.device)
        for kind, ids, c, dofs, x, d in self.parts:
            grad, _ = _grad(kind, x, (0.0,) * self.nd)
            s = torch.bmm(d, torch.bmm(_bmat(grad), self.u[dofs].unsqueeze(2)))[:, :, 0]
            vm[ids] = _von_mises(s)
        return vm

    def nodal(self):
        total, hits = 0.0, torch.zeros(self.n_nodes, dtype=torch.float64, device=self.u.device)
        for kind, ids, c, dofs, x, d in self.parts:
            at = [torch.bmm(d, torch.bmm(_bmat(_grad(kind, x, p)[0]),
                                         self.u[dofs].unsqueeze(2)))[:, :, 0]
                  for p in _points(kind)]
            for a in range(c.shape[1]):
                s = at[0]
                if kind != CPS3:
                    # Gauss values extrapolated to the corner, trilinearly
                    s = sum(v * math.prod(0.5 * (1.0 + math.sqrt(3.0) * math.copysign(1.0, q) * k)
                                          for q, k in zip(p, _CORNERS[kind][a]))
                            for p, v in zip(_points(kind), at))
                if not torch.is_tensor(total):
                    total = torch.zeros(self.n_nodes, s.shape[1], dtype=s.dtype, device=s.device)
                total.index_add_(0, c[:, a], s)
                hits.index_add_(0, c[:, a], torch.ones_like(s[:, 0]))
        return _von_mises(total / hits.clamp_min(1.0)[:, None])

    def reactions(self):
        y = torch.zeros_like(self.u)
        for dofs, ke in self.groups:
            y.index_add_(0, dofs.reshape(-1),
                         torch.bmm(ke, self.u[dofs].unsqueeze(2)).reshape(-1))
        return (y - self.f)[self.fixed]


def _host(t):
    return t.cpu().numpy()


def _exact_conduction(tm):
    dev = _device()
    x = torch.as_tensor(tm.xyz, device=dev)
    c = torch.as_tensor(tm.conn.astype(np.int64), device=dev).reshape(-1, 8)
    k, f = 0.0, torch.zeros(tm.n_nodes, dtype=torch.float64, device=dev)
    corners = torch.tensor(_CORNERS[C3D8], dtype=torch.float64, device=dev)
    for p in _points(C3D8):
        grad, w = _grad(C3D8, x[c], p)
        k = k + torch.bmm(grad, grad.transpose(1, 2)) * (tm.conductivity * w)[:, None, None]
        shape = (1.0 + corners * torch.tensor(p, dtype=torch.float64, device=dev)).prod(1) / 8.0
        f.index_add_(0, c.reshape(-1), (tm.source * w[:, None] * shape).reshape(-1))
    t0 = torch.zeros_like(f)
    node = torch.as_tensor(tm.temp_node, device=dev)
    t0[node] = torch.as_tensor(tm.temp_value, device=dev)
    free = torch.ones_like(f)
    free[node] = 0.0
    lift = torch.zeros_like(f)
    lift.index_add_(0, c.reshape(-1), torch.bmm(k, t0[c].unsqueeze(2)).reshape(-1))
    return _host(t0 + _cg([(c, k)], f - lift, free, None, 1))


def exact(case, seed):
    what = case["what"]
    if not torch.cuda.is_available() and what in ("kept", "serve", "batch"):
        return None  # minutes on host cores
    models = _models(case, seed)
    if what == "conduction":
        return _exact_conduction(models)
    if what == "serve":
        u, vm = [None] * len(models), [None] * len(models)
        for nd in (2, 3):
            at = [k for k, m in enumerate(models) if m.ndof == nd]
            if not at:
                continue
            s = _System([models[k] for k in at])
            un, en = np.cumsum([0] + [models[k].n_dof for k in at]), \
                np.cumsum([0] + [models[k].n_elem for k in at])
            hu, hv = _host(s.u), _host(s.centroid())
            for j, k in enumerate(at):
                u[k], vm[k] = hu[un[j]:un[j + 1]], hv[en[j]:en[j + 1]]
        return {"u": np.concatenate(u), "von_mises": np.concatenate(vm)}
    s = _System(models)
    if what == "kept":
        return {"u": _host(s.u), "cond": None}
    if what == "batch":
        return {"u": _host(s.u), "von_mises": _host(s.centroid())}
    disp = torch.zeros(s.n_nodes, 3, dtype=torch.float64, device=s.u.device)
    disp[:, :s.nd] = s.u.reshape(-1, s.nd)
    return {"u": _host(s.u), "displacements": _host(disp), "von_mises": _host(s.centroid()),
            "nodal_von_mises": _host(s.nodal()), "reactions": _host(s.reactions())}
