"""Workloads of the engine for timing and for comparing two builds of it.

Each case is one call of a user's program through the public entry points of
proxpde_gb300: element assembly on the four element types (`Context.assemble`), the
differentiable diffusion loss (`DiffusionProblem.loss` and its backward), a batch of
small adjoint problems (`batch_adjoint`), a Taylor-Hood Stokes system
(`System.assemble`) and a whole Poisson problem (`Builder` ... `LUSolver.solve`).
`prepare` makes what such a program holds before the call, `run` is the call, and
`exact` computes the same outputs in plain torch, in 64 bits, without the package.

Meshes are unit cubes of n^3 cells (hexahedra, or six Kuhn tetrahedra per cell) with
the interior vertices moved by uniform noise and a log-normal coefficient per element.
"""
import numpy as np
import torch

from proxpde_gb300 import (AssemblyRhsAnalytic, AssemblyStiffnessFE, BCEss, Builder, Context, FESpace, Hexahedron,
                           LUSolver, Mesh, Tetrahedron, side)
from proxpde_gb300 import _lib as L
from proxpde_gb300 import meshgen
from proxpde_gb300.adjoint import DiffusionProblem
from proxpde_gb300.batch import Batch, batch_adjoint

DEV = "cuda"
ETYPE = {"p1": L.P1TET, "p2": L.P2TET, "q1": L.Q1HEX, "q2": L.Q2HEX}
NDOF = {"p1": 4, "p2": 10, "q1": 8, "q2": 27}
LOAD = {"const": L.FN_CONST, "sin3": L.FN_SIN3}
# floating-point operations of one element's stiffness, mass and load, from the
# operation counts of short forms of them (sum factorisation for the hexahedra)
FLOPS = {"p1": 130, "p2": 250, "q1": 1900, "q2": 25000}


# ------------------------------------------------------------------------ the cases
def _assembly(name, et, n, **kw):
    c = {"name": name, "kind": "assembly", "et": et, "n": n, "alpha": 0.2, "sigma": 1.0, "mass": True, "load": "sin3",
         "bc": False, "accumulate": False, "shuffled": False}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest ordinary problem (24,576 tetrahedra): launches and latency count
        _assembly("p1_16", "p1", 16, mass=False, load="const"),
        # a coarse hexahedral mesh as in an inner loop or a unit test, Dirichlet data on
        _assembly("q1_9_bc", "q1", 9, bc=True),
        # an odd-sized mid-size mesh with elements in no particular order (as a mesh
        # generator leaves them), Dirichlet data, added into matrices that hold values
        _assembly("q1_43_shuffled", "q1", 43, bc=True, accumulate=True, shuffled=True),
        # the headline assembly: stiffness, mass and load on 2.1 M hexahedra
        _assembly("q1_128", "q1", 128),
        # linear tetrahedra at size (5.3 M), stiffness, mass and a constant load
        _assembly("p1_96", "p1", 96, load="const"),
        # a small quadratic tetrahedral mesh of odd size, Dirichlet data on
        _assembly("p2_13_bc", "p2", 13, alpha=0.15, sigma=0.5, bc=True),
        # quadratic tetrahedra at size (1.6 M), stiffness and mass
        _assembly("p2_64", "p2", 64, alpha=0.15, sigma=0.5, load="none"),
        # triquadratic hexahedra at size (110,592), stiffness, mass and load
        _assembly("q2_48", "q2", 48),
        # gradient of a PDE-constrained loss with respect to 884,736 coefficients
        {"name": "adjoint_q1_96", "kind": "adjoint", "n": 96},
        # many small adjoint problems of uneven size in one launch
        {"name": "batch_24", "kind": "batch", "nhex": 12, "ntet": 12, "nmin": 8, "nmax": 28},
        # the matrices of a Taylor-Hood Stokes problem
        {"name": "stokes_q2q1_16", "kind": "stokes", "et": "q2", "n": 16},
        # a user's whole Poisson program behind the mesh: build, close, solve
        {"name": "poisson_q1_24", "kind": "poisson", "et": "q1", "n": 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(float(lo) * (float(hi) / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["assembly"] * 8 + ["adjoint", "batch", "stokes", "poisson"])
    if kind == "assembly":
        et = rng.choice(["p1", "p2", "q1", "q2"])
        n = _log_int(rng, *{"p1": (6, 96), "p2": (4, 64), "q1": (6, 128), "q2": (3, 48)}[et])
        c = _assembly("", et, n, alpha=round(rng.uniform(0.05, 0.15 if et[0] == "p" else 0.2), 3),
                      sigma=rng.choice([0.5, 1.0]), mass=rng.random() < 0.75,
                      load=rng.choice(["sin3", "const", "none"]), bc=rng.random() < 0.5,
                      accumulate=rng.random() < 0.3, shuffled=rng.random() < 0.25)
    elif kind == "adjoint":
        c = {"kind": kind, "n": _log_int(rng, 12, 96)}
    elif kind == "batch":
        nmin = rng.randint(8, 14)
        c = {"kind": kind, "nhex": rng.randint(2, 12), "ntet": rng.randint(2, 12), "nmin": nmin,
             "nmax": rng.randint(nmin + 4, 28)}
    elif kind == "stokes":
        et = rng.choice(["q2", "p2"])
        c = {"kind": kind, "et": et, "n": _log_int(rng, 4, 16)}
    else:
        c = {"kind": kind, "et": rng.choice(["q1", "p1"]), "n": _log_int(rng, 6, 24)}
    c.pop("name", None)
    return c


# --------------------------------------------------------------- meshes and numbering
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _lattice(n):
    r = torch.arange(n + 1, device=DEV)
    k, j, i = torch.meshgrid(r, r, r, indexing="ij")
    return torch.stack([i.reshape(-1), j.reshape(-1), k.reshape(-1)], 1)


def _mesh(et, n, alpha, seed, shuffled=False):
    """(lattice indices of the vertices, coordinates, connectivity)"""
    lat = _lattice(n)
    s = [1, n + 1, (n + 1) ** 2]
    cells = (lat[(lat < n).all(1)] * torch.tensor(s, device=DEV)).sum(1)
    if et[0] == "q":
        o = [0, s[0], s[0] + s[1], s[1], s[2], s[0] + s[2], s[0] + s[1] + s[2], s[1] + s[2]]
        off = torch.tensor([o], device=DEV)
    else:
        off = torch.tensor([[0, s[a], s[a] + s[b], s[0] + s[1] + s[2]] for a in range(3) for b in range(3) if a != b],
                           device=DEV)
    conn = (cells[:, None, None] + off[None]).reshape(-1, off.shape[1])
    g = _gen(2 * seed)
    if shuffled:
        conn = conn[torch.randperm(conn.shape[0], generator=g, device=DEV)]
    noise = (torch.rand(lat.shape, generator=g, device=DEV, dtype=torch.float64) * 2 - 1) * (alpha / n)
    interior = ((lat > 0) & (lat < n)).all(1, keepdim=True)
    xyz = lat.to(torch.float64) / n + torch.where(interior, noise, torch.zeros_like(noise))
    return lat, xyz.contiguous(), conn.to(torch.int32).contiguous()


def _coef(ne, sigma, seed):
    return torch.exp(sigma * torch.randn(ne, generator=_gen(2 * seed + 1), device=DEV, dtype=torch.float64))


HEX_EDGES = [(0, 1), (1, 2), (2, 3), (3, 0), (0, 4), (1, 5), (2, 6), (3, 7), (4, 5), (5, 6), (6, 7), (7, 4)]
HEX_FACES = [(0, 3, 2, 1), (3, 0, 4, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (4, 5, 6, 7)]
TET_EDGES = [(0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3)]


def _nodes2(et, lat, conn):
    """Twice the lattice position of every element's nodes: (elements, nodes, 3)."""
    v = lat[conn.long()]
    p = [2 * v]
    if et == "p2":
        p.append(torch.stack([v[:, a] + v[:, b] for a, b in TET_EDGES], 1))
    if et == "q2":
        p.append(torch.stack([v[:, a] + v[:, b] for a, b in HEX_EDGES], 1))
        p.append(torch.stack([v[:, a] + v[:, c] for a, _, c, _ in HEX_FACES], 1))
        p.append((v[:, 0] + v[:, 6])[:, None])
    return torch.cat(p, 1)


def _on_side(p2, n, marker):
    axis, upper = side.PLANE[marker]
    return p2[:, axis] == (2 * n if upper else 0)


WALLS = (side.LEFT, side.BOTTOM, side.BACK, side.RIGHT, side.TOP, side.FRONT)
BCS = ((side.LEFT, 1.0), (side.BOTTOM, -0.5))  # Dirichlet data of the assembly cases: marker, value


# -------------------------------------------------------------------------- prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def run(state):
    return state["run"](state)


def work(case):
    return globals()["_work_" + case["kind"]](case)


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, int(seed))


def _prepare_assembly(c, seed):
    _, xyz, conn = _mesh(c["et"], c["n"], c["alpha"], seed, c["shuffled"])
    ctx = Context(0)
    ctx.set_mesh(ETYPE[c["et"]], xyz, conn)
    ndof, nnz = ctx.build_dofmap(), ctx.build_pattern()
    ctx.set_coef(_coef(conn.shape[0], c["sigma"], seed))
    if c["bc"]:
        ctx.mark_facets_box()
        ctx.set_bc_markers([(m, L.FN_CONST, v) for m, v in BCS])
    bc = 1 if c["bc"] else 0
    st = {"run": _run_assembly, "ctx": ctx, "kw": {
        "op0": {"stiffness": 2, "stiff_coef": 1.0, "apply_bc": bc},
        "vals0": torch.empty(nnz, dtype=torch.float64, device=DEV), "accumulate": c["accumulate"]}}
    if c["mass"]:
        st["kw"].update(op1={"mass": 1, "mass_coef": 1.0, "apply_bc": bc},
                        vals1=torch.empty(nnz, dtype=torch.float64, device=DEV))
    if c["load"] != "none":
        st["kw"]["rhs"] = {"kind": 1, "fn": LOAD[c["load"]], "coef": 1.0, "apply_bc": bc}
    if c["load"] != "none" or c["bc"]:
        st["kw"]["b"] = torch.empty(ndof, dtype=torch.float64, device=DEV)
    st["out"] = [st["kw"][k] for k in ("vals0", "vals1", "b") if k in st["kw"]]
    return st


def _run_assembly(st):
    if st["kw"]["accumulate"]:
        # a time step's matrices: cleared by the program, then added into
        for t in st["out"]:
            t.zero_()
    st["ctx"].assemble(**st["kw"])
    return st["out"]


def _prepare_adjoint(c, seed):
    p = DiffusionProblem.cube_q1(c["n"], seed=1000 + seed)
    log_k = torch.randn(p.nelem, generator=_gen(seed), device=DEV, dtype=torch.float64).requires_grad_(True)
    return {"run": _run_adjoint, "problem": p, "log_k": log_k}


def _run_adjoint(st):
    loss = st["problem"].loss(st["log_k"])
    (grad,) = torch.autograd.grad(loss, st["log_k"])
    return {"loss": loss.detach(), "grad": grad, "u": st["problem"].u}


def _problem_list(c, seed):
    # the sizes belong to the case, the vertices and coefficients to the seed
    sizes = np.random.RandomState(c["nhex"] * 1000 + c["ntet"]).randint(c["nmin"], c["nmax"] + 1, c["nhex"] + c["ntet"])
    r = np.random.RandomState(seed % (1 << 31))
    out = []
    for p, n in enumerate(sizes.tolist()):
        xyz, conn = (meshgen.cube_hex if p < c["nhex"] else meshgen.cube_tet6)(n)
        lat = np.rint(xyz * n)
        interior = ((lat > 0) & (lat < n)).all(1)
        xyz = xyz + np.where(interior[:, None], r.uniform(-0.2 / n, 0.2 / n, xyz.shape), 0.0)
        out.append({"etype": L.Q1HEX if p < c["nhex"] else L.P1TET, "n": n, "xyz": xyz, "conn": conn,
                    "k": np.exp(r.standard_normal(conn.shape[0])), "bc_nodes": np.nonzero(~interior)[0]})
    return out


def _prepare_batch(c, seed):
    probs = _problem_list(c, seed)
    return {"run": _run_batch, "batches": [Batch(probs[:c["nhex"]]), Batch(probs[c["nhex"]:])]}


def _run_batch(st):
    losses, _ = batch_adjoint(st["batches"])
    return {"losses": losses, "grads": [b.grad for b in st["batches"]]}


def _prepare_stokes(c, seed):
    tv, tp = (L.Q2HEX, L.Q1HEX) if c["et"] == "q2" else (L.P2TET, L.P1TET)
    n = c["n"]
    lat, xyz, conn = _mesh(c["et"], n, 0.15, seed)
    cv, cp = Context(0), Context(0)
    for ctx, t in ((cv, tv), (cp, tp)):
        ctx.set_mesh(t, xyz, conn)
        ctx.build_dofmap()
    S = L.System([cv, cp], [3, 1], qr_types=[tv, tv])
    em = torch.from_numpy(cv.get_dofmap().astype(np.int64)).to(DEV)
    d, v = _lid(em, _nodes2(c["et"], lat, conn), n, cv.ndof)
    S.set_bc(0, d.cpu().numpy(), v.cpu().numpy())
    return {"run": _run_stokes, "S": S, "vals": torch.empty(S.nnz, dtype=torch.float64, device=DEV),
            "b": torch.empty(S.ntot, dtype=torch.float64, device=DEV)}


def _lid(em, p2, n, ndof):
    """Walls at rest, lid (top) moving along x: constrained velocity DOFs and values."""
    pos = torch.zeros(ndof, 3, dtype=torch.long, device=DEV)
    pos[em.reshape(-1)] = p2.reshape(-1, 3)
    wall = ((pos == 0) | (pos == 2 * n)).any(1)
    ids = wall.nonzero()[:, 0]
    lid = (pos[ids, 1] == 2 * n).to(torch.float64)
    d = torch.cat([ids + k * ndof for k in range(3)])
    return d, torch.cat([lid, 0 * lid, 0 * lid])


def _run_stokes(st):
    S, vals, b = st["S"], st["vals"], st["b"]
    S.assemble(0, 0, [(L.OP_TENSOR_STIFFNESS, 0.1)], vals, b)
    S.assemble(0, 1, [(L.OP_GRAD, -1.0)], vals, b, accumulate=True)
    S.assemble(1, 0, [(L.OP_DIV, -1.0)], vals, b, accumulate=True)
    return [vals, b]


def _prepare_poisson(c, seed):
    _, xyz, conn = _mesh(c["et"], c["n"], 0.2 if c["et"] == "q1" else 0.15, seed)
    mesh = Mesh(Hexahedron if c["et"] == "q1" else Tetrahedron, xyz.cpu().numpy(), conn.cpu().numpy())
    fe = FESpace(mesh, order=1)
    return {"run": _run_poisson, "fe": fe, "k": _coef(conn.shape[0], 0.5, seed).cpu().numpy(),
            "bcs": [BCEss(fe, m, 0.0) for m in WALLS]}


def _run_poisson(st):
    fe, bcs = st["fe"], st["bcs"]
    builder = Builder(fe)
    builder.buildLhs((AssemblyStiffnessFE(st["k"], fe),), bcs)
    builder.buildRhs((AssemblyRhsAnalytic(L.FN_SIN3, fe),), bcs)
    builder.closeMatrix()
    solver = LUSolver()
    solver.compute(builder)
    return {"indptr": builder.A.indptr, "indices": builder.A.indices, "data": builder.A.data, "b": builder.b,
            "x": solver.solve(builder.b)}


# ----------------------------------------------------------------------------- work
def _sizes(et, n):
    """(elements, vertices, DOFs, entries of the pattern) of a cube, the last about"""
    hexa = et[0] == "q"
    ne, nn = n ** 3 * (1 if hexa else 6), (n + 1) ** 3
    nd = nn if et in ("p1", "q1") else (2 * n + 1) ** 3
    return ne, nn, nd, int(nd * {"p1": 15, "q1": 27, "p2": 28, "q2": 64}[et])


def _work_assembly(c):
    ne, nn, nd, nnz = _sizes(c["et"], c["n"])
    nv, N = (8 if c["et"][0] == "q" else 4), NDOF[c["et"]]
    nmat = 2 if c["mass"] else 1
    b = ne * (4 * nv + 4 * N + 8) + 24 * nn + 8 * nnz * nmat + (8 * nd if c["load"] != "none" or c["bc"] else 0)
    return {"bytes": b, "flops": ne * FLOPS[c["et"]]}


def _cg_work(et, n):
    # two solves of about 3.65 n iterations, each reading the matrix and a few vectors
    ne, _, nd, nnz = _sizes(et, n)
    it = 2 * 3.65 * n
    return np.array([it * (12 * nnz + 72 * nd) + 2 * ne * 80, it * (2 * nnz + 12 * nd) + 2 * ne * FLOPS[et]])


def _work_adjoint(c):
    b, f = _cg_work("q1", c["n"])
    return {"bytes": float(b), "flops": float(f)}


def _work_batch(c):
    mid = (c["nmin"] + c["nmax"]) // 2
    b, f = c["nhex"] * _cg_work("q1", mid) + c["ntet"] * _cg_work("p1", mid)
    return {"bytes": float(b), "flops": float(f)}


def _work_stokes(c):
    ne, nn, nd, nnz = _sizes(c["et"], c["n"])
    N, P = NDOF[c["et"]], (8 if c["et"] == "q2" else 4)
    _, _, ndp, _ = _sizes("q1" if c["et"] == "q2" else "p1", c["n"])
    # nine velocity blocks, the six couplings (about P/N of a block's entries each)
    out = 8 * (9 * nnz + 6 * nnz * P // N) + 8 * (3 * nd + ndp)
    return {"bytes": ne * 4 * (2 * P + N) + 24 * nn + out, "flops": ne * 3 * FLOPS[c["et"]]}


def _work_poisson(c):
    ne, nn, nd, nnz = _sizes(c["et"], c["n"])
    b, f = _cg_work(c["et"], c["n"])
    return {"bytes": float(b) + 24 * nnz, "flops": float(f)}


# ---------------------------------------------------------------------------- exact
def _rule(et):
    """Quadrature points and weights (src/qr.cpp:199-320)."""
    f = lambda a: torch.tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
    if et == "p1":
        a, b = 0.1381966011250105, 0.5854101966249685
        return f([[a, a, a], [b, a, a], [a, b, a], [a, a, b]]), f([0.25 / 6] * 4)
    if et == "p2":
        c1, c2, d1, d2 = 0.0714285714285714, 0.7857142857142857, 0.399403576166799, 0.100596423833201
        p = [[.25] * 3, [c1, c1, c1], [c2, c1, c1], [c1, c2, c1], [c1, c1, c2], [d1, d1, d2], [d1, d2, d1],
             [d2, d1, d1], [d1, d2, d2], [d2, d1, d2], [d2, d2, d1]]
        return f(p), f([-0.0131555555555556] + [0.0076222222222222] * 4 + [0.024888888888889] * 6)
    if et == "q1":
        x, w = [-0.5773502691896258, 0.5773502691896258], [1.0, 1.0]
    else:
        x, w = [-0.774596669241483, 0.0, 0.774596669241483], [5.0 / 9, 8.0 / 9, 5.0 / 9]
    r = range(len(x))
    return (f([[x[i], x[j], x[k]] for k in r for j in r for i in r]), f([w[i] * w[j] * w[k] for k in r for j in r for i in r]))


Q1IDX = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
Q2IDX = Q1IDX + [(2, 0, 0), (1, 2, 0), (2, 1, 0), (0, 2, 0), (0, 0, 2), (1, 0, 2), (1, 1, 2), (0, 1, 2), (2, 0, 1),
                 (1, 2, 1), (2, 1, 1), (0, 2, 1), (2, 2, 0), (0, 2, 2), (2, 0, 2), (1, 2, 2), (2, 1, 2), (2, 2, 1),
                 (2, 2, 2)]


def _shape(et, p):
    """(values (nq, N), gradients (nq, N, 3)) of the reference basis at the points p"""
    x, y, z = p[:, 0], p[:, 1], p[:, 2]
    one, zero = torch.ones_like(x), torch.zeros_like(x)
    if et[0] == "p":
        lam = [1 - x - y - z, x, y, z]
        dl = [[-one, -one, -one], [one, zero, zero], [zero, one, zero], [zero, zero, one]]
        if et == "p1":
            return torch.stack(lam, 1), torch.stack([torch.stack(d, 1) for d in dl], 1)
        phi = [v * (2 * v - 1) for v in lam] + [4 * lam[a] * lam[b] for a, b in TET_EDGES]
        d = [[(4 * lam[a] - 1) * dl[a][k] for k in range(3)] for a in range(4)]
        d += [[4 * (lam[a] * dl[b][k] + lam[b] * dl[a][k]) for k in range(3)] for a, b in TET_EDGES]
        return torch.stack(phi, 1), torch.stack([torch.stack(v, 1) for v in d], 1)
    if et == "q1":
        f = [[0.5 * (1 - t), 0.5 * (1 + t)] for t in (x, y, z)]
        g = [[-0.5 * one, 0.5 * one]] * 3
        idx = Q1IDX
    else:
        f = [[0.5 * t * (t - 1), 0.5 * t * (t + 1), 1 - t * t] for t in (x, y, z)]
        g = [[t - 0.5, t + 0.5, -2 * t] for t in (x, y, z)]
        idx = Q2IDX
    phi = [f[0][a] * f[1][b] * f[2][c] for a, b, c in idx]
    d = [[g[0][a] * f[1][b] * f[2][c], f[0][a] * g[1][b] * f[2][c], f[0][a] * f[1][b] * g[2][c]] for a, b, c in idx]
    return torch.stack(phi, 1), torch.stack([torch.stack(v, 1) for v in d], 1)


def _numbering(et, lat, conn, n):
    """First-touch DOF map (include/dof.hpp:111-329) and twice the lattice positions."""
    p2 = _nodes2(et, lat, conn)
    m = 2 * n + 1
    key = ((p2[..., 0] * m + p2[..., 1]) * m + p2[..., 2]).reshape(-1)
    uniq, inv = torch.unique(key, return_inverse=True)
    first = torch.full((uniq.numel(),), key.numel(), dtype=torch.long, device=DEV)
    first.scatter_reduce_(0, inv, torch.arange(key.numel(), device=DEV), "amin")
    ids = torch.empty_like(uniq)
    ids[torch.argsort(first)] = torch.arange(uniq.numel(), device=DEV)
    em = ids[inv].reshape(p2.shape[:2])
    pos = torch.zeros(uniq.numel(), 3, dtype=torch.long, device=DEV)
    pos[em.reshape(-1)] = p2.reshape(-1, 3)
    return em, pos


def _geometry(et, X, pts):
    """J^-1 (row: reference direction), |det J| and the quadrature points of CurFE."""
    _, dv = _shape("q1" if et[0] == "q" else "p1", pts)
    J = torch.einsum("enr,qnd->eqrd", X - X[:, :1], dv)
    a, b, c = J[..., 0], J[..., 1], J[..., 2]
    adj = torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], -2)
    det = (a * adj[..., 0, :]).sum(-1)
    origin = X.mean(1) if et[0] == "q" else X[:, 0]
    return adj / det[..., None, None], det.abs(), origin[:, None] + torch.einsum("eqrd,qd->eqr", J, pts)


def _chunks(ne, N):
    step = max(1, 40_000_000 // (N * N * 3))
    return [(s, min(ne, s + step)) for s in range(0, ne, step)]


def _load(fn, qp):
    return torch.ones_like(qp[..., 0]) if fn == "const" else torch.sin(np.pi * qp).prod(-1)


def _elements(et, xyz, conn, k, mass, load):
    """Element matrices and loads, by quadrature."""
    pts, w = _rule(et)
    phi, dphi = _shape(et, pts)
    N = NDOF[et]
    for s, t in _chunks(conn.shape[0], N):
        Ji, det, qp = _geometry(et, xyz[conn[s:t].long()], pts)
        D = torch.einsum("qnd,eqdr->enqr", dphi, Ji)
        wd = det * w
        Dw = (D * (wd * k[s:t, None])[:, None, :, None]).reshape(t - s, N, -1)
        K = Dw @ D.reshape(t - s, N, -1).transpose(1, 2)
        M = torch.einsum("eq,qi,qj->eij", wd, phi, phi) if mass else None
        F = (wd * _load(load, qp)) @ phi if load != "none" else None
        yield s, t, K, M, F


def _pattern(em, ndof):
    key = (em[:, :, None] * ndof + em[:, None, :]).reshape(-1)
    uniq, inv = torch.unique(key, return_inverse=True)
    return uniq, inv.reshape(em.shape[0], em.shape[1], em.shape[1])


def _assemble(et, xyz, conn, em, ndof, k, mass, load, cmask=None, cval=None, need_b=True):
    """(entry keys, K, M, b), condensed on both matrices where cmask is given."""
    uniq, inv = _pattern(em, ndof)
    K = torch.zeros(uniq.numel(), dtype=torch.float64, device=DEV)
    M = torch.zeros_like(K) if mass else None
    b = torch.zeros(ndof, dtype=torch.float64, device=DEV)
    for s, t, Ke, Me, Fe in _elements(et, xyz, conn, k, mass, load):
        dofs = em[s:t]
        c = cmask[dofs] if cmask is not None else None
        if Fe is not None:
            b.index_add_(0, dofs.reshape(-1), (Fe if c is None else Fe * ~c).reshape(-1))
        for out, E in ((K, Ke), (M, Me)):
            if E is None:
                continue
            if c is not None:
                h = torch.where(c, cval[dofs], torch.zeros_like(cval[dofs]))
                f = torch.where(c, h, -(E @ h[:, :, None])[:, :, 0])
                b.index_add_(0, dofs.reshape(-1), f.reshape(-1))
                E = torch.where(c[:, :, None] | c[:, None, :], torch.zeros_like(E), E) + torch.diag_embed(c.to(E))
            out.index_add_(0, inv[s:t].reshape(-1), E.reshape(-1))
    return uniq, K, M, b


def _exact_assembly(c, seed):
    lat, xyz, conn = _mesh(c["et"], c["n"], c["alpha"], seed, c["shuffled"])
    em, pos = _numbering(c["et"], lat, conn, c["n"])
    ndof = pos.shape[0]
    mask = val = None
    if c["bc"]:
        mask = torch.zeros(ndof, dtype=torch.bool, device=DEV)
        val = torch.zeros(ndof, dtype=torch.float64, device=DEV)
        for m, v in BCS:
            on = _on_side(pos, c["n"], m)
            mask |= on
            val[on] = v
    _, K, M, b = _assemble(c["et"], xyz, conn, em, ndof, _coef(conn.shape[0], c["sigma"], seed), c["mass"], c["load"],
                           mask, val)
    out = [K] + ([M] if c["mass"] else [])
    return out + ([b] if c["load"] != "none" or c["bc"] else [])


def _csr(uniq, vals, ndof):
    rows = torch.div(uniq, ndof, rounding_mode="floor")
    ptr = torch.zeros(ndof + 1, dtype=torch.long, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=ndof), 0)
    return torch.sparse_csr_tensor(ptr, uniq - rows * ndof, vals, (ndof, ndof)), rows, uniq - rows * ndof


def _solve(A, diag, b, tol=1e-14):
    """Jacobi-preconditioned conjugate gradients to a residual far below the engine's."""
    x = torch.zeros_like(b)
    r, z = b.clone(), b / diag
    p, rz, stop = z.clone(), b @ z, tol * torch.linalg.norm(b)
    for it in range(20000):
        q = A @ p
        al = rz / (p @ q)
        x += al * p
        r -= al * q
        if it % 16 == 15 and torch.linalg.norm(r) <= stop:
            break
        z = r / diag
        new = r @ z
        p = z + (new / rz) * p
        rz = new
    return x


def _adjoint(et, lat, xyz, conn, n, k):
    """(loss, gradient with respect to log k, u) of 1/2 |u - sin3|_M^2, K(k) u = 1"""
    em, pos = _numbering(et, lat, conn, n)
    ndof = pos.shape[0]
    mask = ((pos == 0) | (pos == 2 * n)).any(1)
    zero = torch.zeros(ndof, dtype=torch.float64, device=DEV)
    X = torch.zeros(ndof, 3, dtype=torch.float64, device=DEV)
    X[em.reshape(-1)] = xyz[conn.long()].reshape(-1, 3)
    uniq, K, _, b = _assemble(et, xyz, conn, em, ndof, k, False, "const", mask, zero)
    _, _, M, _ = _assemble(et, xyz, conn, em, ndof, k, True, "none")
    A, rows, cols = _csr(uniq, K, ndof)
    diag = torch.zeros_like(zero)
    diag[rows[rows == cols]] = K[rows == cols]
    u = _solve(A, diag, b)
    w = u - torch.sin(np.pi * X).prod(1)
    Mw = _csr(uniq, M, ndof)[0] @ w
    lam = _solve(A, diag, Mw)
    free = (~mask).to(torch.float64)
    uf, lf = u * free, lam * free
    g = torch.empty(conn.shape[0], dtype=torch.float64, device=DEV)
    for s, t, Ke, _, _ in _elements(et, xyz, conn, k, False, "none"):
        g[s:t] = -torch.einsum("ei,eij,ej->e", uf[em[s:t]], Ke, lf[em[s:t]])
    return 0.5 * (w @ Mw), g, u


def _exact_adjoint(c, seed):
    n = c["n"]
    xyz, conn = meshgen.cube_hex(n)
    xyz = torch.from_numpy(meshgen.perturb(xyz, n, 0.2, 1000 + seed)).to(DEV)
    conn = torch.from_numpy(conn.astype(np.int32)).to(DEV)
    log_k = torch.randn(conn.shape[0], generator=_gen(seed), device=DEV, dtype=torch.float64)
    J, g, u = _adjoint("q1", _lattice(n), xyz, conn, n, torch.exp(log_k))
    return {"loss": J, "grad": g, "u": u}


def _exact_batch(c, seed):
    losses, grads = [], [[], []]
    for p in _problem_list(c, seed):
        hexa = p["etype"] == L.Q1HEX
        J, g, _ = _adjoint("q1" if hexa else "p1", _lattice(p["n"]), torch.from_numpy(p["xyz"]).to(DEV),
                           torch.from_numpy(p["conn"].astype(np.int32)).to(DEV), p["n"],
                           torch.from_numpy(p["k"]).to(DEV))
        losses.append(float(J))
        grads[0 if hexa else 1].append(g)
    return {"losses": np.array(losses), "grads": [torch.cat(g) for g in grads]}


def _exact_stokes(c, seed):
    n, ev = c["n"], c["et"]
    ep = "q1" if ev == "q2" else "p1"
    lat, xyz, conn = _mesh(ev, n, 0.15, seed)
    (emv, posv), (emp, posp) = _numbering(ev, lat, conn, n), _numbering(ep, lat, conn, n)
    nv, npr = posv.shape[0], posp.shape[0]
    ntot = 3 * nv + npr
    pts, w = _rule(ev)
    phv, dpv = _shape(ev, pts)
    php, _ = _shape(ep, pts)
    Nv, Np = phv.shape[1], php.shape[1]
    dofs = torch.cat([emv, emv + nv, emv + 2 * nv, emp + 3 * nv], 1)
    uniq, inv = _pattern(dofs, ntot)
    d, v = _lid(emv, _nodes2(ev, lat, conn), n, nv)
    mask = torch.zeros(ntot, dtype=torch.bool, device=DEV)
    val = torch.zeros(ntot, dtype=torch.float64, device=DEV)
    mask[d] = True
    val[d] = v
    vals = torch.zeros(uniq.numel(), dtype=torch.float64, device=DEV)
    b = torch.zeros(ntot, dtype=torch.float64, device=DEV)
    for s, t in _chunks(conn.shape[0], 3 * Nv + Np):
        Ji, det, _ = _geometry(ev, xyz[conn[s:t].long()], pts)
        D = torch.einsum("qnd,eqdr->eqnr", dpv, Ji)
        wd = det * w
        B = torch.einsum("eqia,eqjb->eaibj", D * wd[:, :, None, None], D)
        lap = B[:, 0, :, 0] + B[:, 1, :, 1] + B[:, 2, :, 2]
        E = torch.zeros(t - s, 3 * Nv + Np, 3 * Nv + Np, dtype=torch.float64, device=DEV)
        G = torch.einsum("eqia,eqj->eaij", D * wd[:, :, None, None], php.expand(t - s, -1, -1))
        for a in range(3):
            ra = slice(a * Nv, (a + 1) * Nv)
            for e in range(3):
                E[:, ra, e * Nv:(e + 1) * Nv] = 0.1 * (B[:, a, :, e] + (lap if a == e else 0))
            E[:, ra, 3 * Nv:] = -G[:, a]
            E[:, 3 * Nv:, ra] = -G[:, a].transpose(1, 2)
        dd = dofs[s:t]
        cm = mask[dd]
        h = val[dd] * cm
        f = torch.where(cm, h, -(E @ h[:, :, None])[:, :, 0])
        b.index_add_(0, dd.reshape(-1), f.reshape(-1))
        E = torch.where(cm[:, :, None] | cm[:, None, :], torch.zeros_like(E), E) + torch.diag_embed(cm.to(E))
        vals.index_add_(0, inv[s:t].reshape(-1), E.reshape(-1))
    return [vals, b]


def _exact_poisson(c, seed):
    et, n = c["et"], c["n"]
    lat, xyz, conn = _mesh(et, n, 0.2 if et == "q1" else 0.15, seed)
    em, pos = _numbering(et, lat, conn, n)
    ndof = pos.shape[0]
    mask = ((pos == 0) | (pos == 2 * n)).any(1)
    uniq, K, _, b = _assemble(et, xyz, conn, em, ndof, _coef(conn.shape[0], 0.5, seed), False, "sin3", mask,
                              torch.zeros(ndof, dtype=torch.float64, device=DEV))
    keep = K.abs() > 1e-16
    A, rows, cols = _csr(uniq[keep], K[keep], ndof)
    diag = torch.zeros_like(b)
    diag[rows[rows == cols]] = K[keep][rows == cols]
    return {"indptr": None, "indices": None, "data": K[keep], "b": b, "x": _solve(A, diag, b, 1e-15)}
