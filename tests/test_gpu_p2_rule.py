"""P2 matrices of calls with one matrix, both in one operator, mass before stiffness or Dirichlet
conditions, one element at a time, against the 11-point rule in long double: its points and weights have
13 to 16 digits, so that the matrices differ by up to 2.4e-15 (norm; mass 8e-16) from the exact moments."""
import numpy as np
import pytest

import oracle as O
from helpers import gpu_assemble

pytestmark = pytest.mark.gpu

K_OP = {"stiffness": 2, "stiff_coef": 1.0}
M_OP = {"mass": 1, "mass_coef": 1.0}
N = 128


def reference(d, k):
    """(N, 10, 10) stiffness and mass by the rule"""
    f = np.longdouble
    c1, c2, d1, d2 = f(0.0714285714285714), f(0.7857142857142857), f(0.399403576166799), f(0.100596423833201)
    p = np.array([[f(0.25)] * 3, [c1, c1, c1], [c2, c1, c1], [c1, c2, c1], [c1, c1, c2], [d1, d1, d2], [d1, d2, d1],
                  [d2, d1, d1], [d1, d2, d2], [d2, d1, d2], [d2, d2, d1]], dtype=f)
    w = np.array([-0.0131555555555556] + [0.0076222222222222] * 4 + [0.024888888888889] * 6, dtype=f)
    lam = np.concatenate([1 - p.sum(axis=1, keepdims=True), p], axis=1)
    dl = np.concatenate([-np.ones((1, 3)), np.eye(3)]).astype(f)
    edges = [(0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3)]
    phi = np.concatenate([lam * (2 * lam - 1), np.stack([4 * lam[:, a] * lam[:, c] for a, c in edges], axis=1)], axis=1)
    g = np.concatenate([(4 * lam - 1)[:, :, None] * dl, np.stack(
        [4 * (lam[:, a, None] * dl[c] + lam[:, c, None] * dl[a]) for a, c in edges], axis=1)], axis=1)  # (q, i, 3)
    D = d.astype(f)
    C = np.stack([np.cross(D[:, 1], D[:, 2]), np.cross(D[:, 2], D[:, 0]), np.cross(D[:, 0], D[:, 1])], axis=1)
    det = np.abs((D[:, 0] * C[:, 0]).sum(axis=1))
    G = np.einsum("qik,ekr->eqir", g, C)
    K = np.einsum("q,eqir,eqjr->eij", w, G, G) * (k / det)[:, None, None]
    return K, np.einsum("q,qi,qj->ij", w, phi, phi) * det[:, None, None]


@pytest.mark.parametrize("ops,bc", [([K_OP], 0), ([M_OP], 0), ([M_OP, K_OP], 0),
                                    ([{"stiffness": 2, "stiff_coef": 1.0, "mass": 1, "mass_coef": 1.0}], 0),
                                    ([K_OP, M_OP], 1)], ids=["K", "M", "M, K", "K+M", "K, M bc"])
@pytest.mark.parametrize("scatter", [0, 1], ids=["reduce", "colour"])
def test_matrices_are_the_rule_s(engine, ops, bc, scatter):
    r = np.random.RandomState(4)
    d = np.triu(np.ones((3, 3))).T + r.uniform(-0.2, 0.2, (N, 3, 3))
    d = np.rint(d * 2.0 ** 20) / 2.0 ** 20  # cofactors and determinant need no more than 63 bits
    xyz = np.concatenate([np.zeros((N, 1, 3)), d], axis=1).reshape(-1, 3)
    conn = np.arange(4 * N, dtype=np.uint32).reshape(N, 4)
    k = np.exp(r.standard_normal(N))
    em, ndof = O.dofmap(O.P2TET, 4 * N, conn)
    ids = em[::2, 0].astype(np.uint32)  # vertex 0 of every other element: every warp has some
    g = gpu_assemble(O.P2TET, xyz, conn, [dict(o, apply_bc=bc) for o in ops], k=k, scatter=scatter,
                     bc=(ids, np.zeros(ids.size)) if bc else None)
    K, M = reference(d, k)
    e = em.astype(np.int64)
    for op, v in zip(ops, g["struct_vals"]):
        ref = (K if op.get("stiffness") else 0) + (M if op.get("mass") else 0)
        rp, ci = g["pattern"][0], g["pattern"][1]
        A = np.zeros((N, 10, 10))
        for n in range(N):
            for i in range(10):
                row = slice(rp[e[n, i]], rp[e[n, i] + 1])
                A[n, i] = v[row][np.searchsorted(ci[row], e[n])]
        s = slice(1, 10) if bc else slice(0, 10)  # without the constrained node
        err = (A - ref)[:, s, s]
        err, ref = np.sqrt((err ** 2).sum(axis=(1, 2))), np.sqrt((ref ** 2).sum(axis=(1, 2)))
        # six products and additions an entry, each within half an ulp of the element's norm at most, and the
        # tensors' own rounding (eleven terms, summed in FP64)
        assert (err / ref).max() <= 6 * 2.0 ** -53


def test_autotune_times_the_group_kernel_once(engine):
    """The group kernel has one block size: its three candidates are one launch and one time, and the first of
    them is kept unless a colouring is faster."""
    from proxpde_gb300 import Context
    from helpers import problem

    xyz, conn, k = problem("tet6", 6, 0.15, seed=4, sigma=1.0)
    ctx = Context(0)
    ctx.set_mesh(O.P2TET, xyz, conn)
    ctx.build_dofmap()
    ctx.build_pattern()
    ctx.set_coef(k)
    rep = ctx.autotune(op0=K_OP, op1=M_OP)
    ms = [c[2] for c in rep["candidates"] if c[1] == "reduce"]
    assert len(ms) == 3 and len(set(ms)) == 1
    assert rep["scatter"] != "reduce" or rep["threads"] == rep["candidates"][0][0]
