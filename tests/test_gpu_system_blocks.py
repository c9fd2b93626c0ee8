"""The component blocks of a vector space (one position search per node pair, sums of Q2 in 64-bit fixed
point): positions with other spaces before and behind them and conditions on some components, against the
oracle's per-entry triplets; and the values of Q2 elements of strongly different shapes, one element at a
time, against long double, every entry held to the geometric mean of its two diagonal entries."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle as O
from helpers import assert_close, compare_csr, problem

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

LAYOUTS = [[(3, "v")], [(3, "v"), (1, "p")], [(1, "p"), (3, "v")], [(2, "v"), (2, "v")], [(1, "v"), (3, "v"), (2, "p")]]


@pytest.mark.parametrize("layout", LAYOUTS, ids=["+".join(f"{d}{k}" for d, k in s) for s in LAYOUTS])
@pytest.mark.parametrize("tv,tp,gen", [(O.Q2HEX, O.Q1HEX, "hex"), (O.P2TET, O.P1TET, "tet6")], ids=["q2", "p2"])
def test_positions(engine, tv, tp, gen, layout):
    from proxpde_gb300 import Context
    from proxpde_gb300._lib import OP_MASS, OP_STIFFNESS, OP_TENSOR_STIFFNESS, System

    xyz, conn, _ = problem(gen, 2, 0.15, seed=3)
    spaces, ctxs, off = [], [], 0
    for dim, kind in layout:
        t = tv if kind == "v" else tp
        em, nd = O.dofmap(t, xyz.shape[0], conn)
        spaces.append(dict(t=t, qr=tv, dim=dim, offset=off, ndof=nd, em=em))
        off += dim * nd
        c = Context(0)
        c.set_mesh(t, xyz, conn)
        c.build_dofmap()
        ctxs.append(c)
    S_o = O.System(xyz, conn, spaces, off)
    S = System(ctxs, [d for d, _ in layout], qr_types=[tv] * len(layout))
    assert S.ntot == off
    for s, sp_ in enumerate(spaces):
        n = sp_["dim"] * sp_["ndof"]
        dofs = np.arange(s, n, 5)  # all components, every element some
        vals = np.cos(np.arange(dofs.size))
        mask, mv = np.zeros(n, np.uint8), np.zeros(n)
        mask[dofs], mv[dofs] = 1, vals
        S_o.set_bc(s, mask, mv, 2.0)
        S.set_bc(s, dofs, vals, 2.0)
    v = torch.zeros(S.nnz, dtype=torch.float64, device="cuda:0")
    b = torch.zeros(S.ntot, dtype=torch.float64, device="cuda:0")
    for s, (dim, _) in enumerate(layout):
        ops = [(O.STIFF, 2.0), (O.MASS, 0.5)] + ([(O.TENSOR_STIFF, 0.1)] if dim == 3 else [])
        dev = {O.STIFF: OP_STIFFNESS, O.MASS: OP_MASS, O.TENSOR_STIFF: OP_TENSOR_STIFFNESS}
        S_o.call(s, s, ops)
        S.assemble(s, s, [(dev[k], c) for k, c in ops], v, b, accumulate=True)
    csr = S_o.close()
    rp, ci = S.get_pattern()
    A = sp.csr_matrix((v.cpu().numpy(), ci, rp), shape=(S.ntot, S.ntot))
    A.data[np.abs(A.data) <= 1e-16] = 0.0
    A.eliminate_zeros()
    A.sort_indices()
    compare_csr((A.indptr, A.indices, A.data), csr, S.ntot, what="system blocks")
    assert_close(b.cpu().numpy(), S_o.b, what="system blocks b")


IDX = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1), (2, 0, 0), (1, 2, 0),
       (2, 1, 0), (0, 2, 0), (0, 0, 2), (1, 0, 2), (1, 1, 2), (0, 1, 2), (2, 0, 1), (1, 2, 1), (2, 1, 1), (0, 2, 1),
       (2, 2, 0), (0, 2, 2), (2, 0, 2), (1, 2, 2), (2, 1, 2), (2, 2, 1), (2, 2, 2)]


def reference(X):
    """B[e, c, d, i, j] = int grad_c phi_i grad_d phi_j of Q2 on the hexahedra X (E, 8, 3), and the condition
    max_q | |J^-1| |J| | of their Jacobians, in long double"""
    f = np.longdouble
    t = f(0.774596669241483)
    x1, w1 = np.array([-t, 0, t], f), np.array([f(5) / 9, f(8) / 9, f(5) / 9])
    q = np.array([(a, b, c) for a in range(3) for b in range(3) for c in range(3)])
    p, w = x1[q], w1[q].prod(axis=1)
    l = np.stack([p * (p - 1) / 2, p * (p + 1) / 2, 1 - p * p])
    d = np.stack([p - f(0.5), p + f(0.5), -2 * p])
    g = np.empty((27, 27, 3), f)
    for n, i in enumerate(IDX):
        for c in range(3):
            g[:, n, c] = np.prod([(d if a == c else l)[i[a]][:, a] for a in range(3)], axis=0)
    sg = np.array([[2 * k - 1 for k in IDX[v]] for v in range(8)], f)
    dv = np.empty((27, 8, 3), f)
    for c in range(3):
        o = [a for a in range(3) if a != c]
        dv[:, :, c] = sg[:, c] * (1 + p[:, None, o[0]] * sg[:, o[0]]) * (1 + p[:, None, o[1]] * sg[:, o[1]]) / 8
    J = np.einsum("evr,qvc->eqrc", X.astype(f), dv)
    C = np.stack([np.cross(J[..., 1], J[..., 2]), np.cross(J[..., 2], J[..., 0]), np.cross(J[..., 0], J[..., 1])], axis=2)
    det = (J[..., 0] * C[:, :, 0]).sum(axis=2)
    Ji = C / det[..., None, None]
    cond = np.abs(np.einsum("eqkr,eqrc->eqkc", np.abs(Ji), np.abs(J))).sum(axis=3).max(axis=(1, 2))
    # terms of a Jacobian entry against the entry: eight vertices
    D = np.einsum("qnk,eqkr->eqnr", g, Ji)
    return np.einsum("eq,eqic,eqjd->ecdij", np.abs(det) * w, D, D, optimize=True), cond.astype(float)


@pytest.mark.parametrize("shape", ["cube", "thin", "thin rotated", "shear", "needle", "wedge"])
def test_q2_values_entrywise(engine, shape):
    from proxpde_gb300 import Context
    from proxpde_gb300._lib import OP_STIFFNESS, OP_TENSOR_STIFFNESS, System

    r = np.random.RandomState(5)
    E = 12
    corner = np.array([IDX[v] for v in range(8)], float)
    Xe = corner + r.uniform(-0.1, 0.1, (E, 8, 3))
    if shape in ("thin", "thin rotated"):
        Xe = Xe * [1.0, 1.0, 0.01]
    elif shape == "needle":
        Xe = Xe * [1.0, 0.01, 0.01]
    elif shape == "shear":
        Xe = Xe @ np.array([[1.0, 0.0, 0.0], [1.0, 0.02, 0.0], [0.3, 0.2, 1.0]])
    elif shape == "wedge":
        Xe[:, :, 0] *= 0.02 + Xe[:, :, 2].clip(0.0)
    if shape == "thin rotated":
        Q, _ = np.linalg.qr(r.standard_normal((3, 3)))
        Xe = Xe @ Q
    Xe = Xe - Xe[:, :1]
    xyz = np.ascontiguousarray(Xe.reshape(-1, 3))
    conn = np.arange(8 * E, dtype=np.uint32).reshape(E, 8)
    c = Context(0)
    c.set_mesh(O.Q2HEX, xyz, conn)
    nd = c.build_dofmap()
    em = c.get_dofmap().astype(np.int64)
    S = System([c], [3])
    rp, ci = S.get_pattern()
    v = torch.zeros(S.nnz, dtype=torch.float64, device="cuda:0")
    b = torch.zeros(S.ntot, dtype=torch.float64, device="cuda:0")
    B, cond = reference(Xe)
    K = np.einsum("eccij->eij", B)
    for ops, want in (([(OP_STIFFNESS, 1.0)], lambda c1, c2: K if c1 == c2 else 0 * K),
                      ([(OP_TENSOR_STIFFNESS, 1.0)], lambda c1, c2: B[:, c1, c2] + (K if c1 == c2 else 0))):
        S.assemble(0, 0, ops, v, b)
        A = sp.csr_matrix((v.cpu().numpy(), ci, rp), shape=(S.ntot, S.ntot))
        for e in range(E):
            dofs = np.concatenate([em[e] + k * nd for k in range(3)])
            a = A[dofs][:, dofs].toarray()
            ref = np.block([[want(c1, c2)[e].astype(float) for c2 in range(3)] for c1 in range(3)])
            err = np.abs(a - np.block([[want(c1, c2)[e] for c2 in range(3)] for c1 in range(3)]))
            dia = np.sqrt(np.diag(ref))
            # the Jacobian's sums of eight terms, its inverse (both times the condition, twice as the gradients
            # enter twice), three products a gradient, 27 points and the trace
            tol = (2 * (8 + 12) * cond[e] + 2 * 4 + 27 + 3) * 2.0 ** -53
            assert (err / np.outer(dia, dia)).max() <= tol
