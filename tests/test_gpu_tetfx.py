"""The fixed-point parts of the tetrahedra: P1 stiffness (csrc/pxg_assemble.cu, p1Fixed), the
sine load of P1 and P2 (csrc/pxg_tetload.cu) and the two-warp group kernel of P2 with
Dirichlet conditions and single matrices (csrc/pxg_p2group.cu), at partial groups and
blocks, units and shapes of every kind, against the oracle under the rule of helpers.py."""
import numpy as np
import pytest

import oracle as O
from helpers import assert_close, compare_csr, gpu_assemble, oracle_lhs, problem

pytestmark = pytest.mark.gpu

K_OP = {"stiffness": 2, "stiff_coef": 1.0, "apply_bc": 0}
M_OP = {"mass": 1, "mass_coef": 1.0, "apply_bc": 0}
SIN3 = {"kind": 1, "fn": O.FN_SIN3, "coef": 1.0, "apply_bc": 0}


def check_long_double(t, xyz, conn, k):
    """K(k) of P1 and the sine load of P1 and P2 in numpy's long double (64-bit or longer
    significand): the oracle's J and Gram determinant lose about the square of an element's
    aspect ratio (2e-11 at 1:100), more than the tolerance."""
    f = np.longdouble
    em, ndof = O.dofmap(t, xyz.shape[0], conn)
    g = gpu_assemble(t, xyz, conn, [K_OP], rhs=SIN3, k=k)
    X = xyz[conn.astype(np.int64)].astype(f)
    D = X[:, 1:] - X[:, :1]
    C = np.stack([np.cross(D[:, 1], D[:, 2]), np.cross(D[:, 2], D[:, 0]), np.cross(D[:, 0], D[:, 1])], axis=1)
    det = np.abs((D[:, 0] * C[:, 0]).sum(axis=1))
    e = em.astype(np.int64)
    if t == O.P1TET:
        p = np.full((4, 3), f(0.1381966011250105)) + (f(0.5854101966249685) - f(0.1381966011250105)) * np.eye(4, 3, -1)
        w = np.full(4, f(0.25 / 6))
        phi = np.concatenate([1 - p.sum(axis=1, keepdims=True), p], axis=1)
        A = np.concatenate([-C.sum(axis=1)[:, None], C], axis=1)
        K = np.zeros((ndof, ndof), f)
        np.add.at(K, (e[:, :, None], e[:, None, :]), np.einsum("eir,ejr->eij", A, A) * (k / det / 6)[:, None, None])
        rp, ci, v = g["mats"][0]
        rows = np.repeat(np.arange(ndof), np.diff(rp))
        o = (rp, ci, K[rows, ci].astype(np.float64))
        assert compare_csr((rp, ci, v), o, ndof, what="tet fixed point flat") == 0
    else:
        c1, c2, d1, d2 = f(0.0714285714285714), f(0.7857142857142857), f(0.399403576166799), f(0.100596423833201)
        p = np.array([[f(0.25)] * 3, [c1, c1, c1], [c2, c1, c1], [c1, c2, c1], [c1, c1, c2], [d1, d1, d2], [d1, d2, d1],
                      [d2, d1, d1], [d1, d2, d2], [d2, d1, d2], [d2, d2, d1]], dtype=f)
        w = np.array([-0.0131555555555556] + [0.0076222222222222] * 4 + [0.024888888888889] * 6, dtype=f)
        lam = np.concatenate([1 - p.sum(axis=1, keepdims=True), p], axis=1)
        edges = [(0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3)]
        phi = np.concatenate([lam * (2 * lam - 1), np.stack([4 * lam[:, a] * lam[:, c] for a, c in edges], axis=1)], axis=1)
    fq = np.sin(f(np.pi) * (X[:, :1] + np.einsum("qa,ear->eqr", p, D))).prod(axis=2)
    b = np.zeros(ndof, f)
    np.add.at(b, e, (det[:, None] * w * fq) @ phi)
    assert_close(g["b"], b.astype(np.float64), what="tet fixed point flat b")


def check(t, xyz, conn, k, ops, rhs=None, bc=False):
    em, ndof = O.dofmap(t, xyz.shape[0], conn)
    mask = val = pair = None
    if bc:
        x = O.dof_coords(t, xyz, conn, em, ndof)
        mask = O.plane_bc_mask(x, [("x", x[:, 0].min())])
        ids = np.nonzero(mask)[0]
        val = np.where(mask, np.sin(np.arange(ndof)), 0.0)
        pair = (ids.astype(np.uint32), val[ids])
        ops = [dict(o, apply_bc=1) for o in ops]
        rhs = dict(rhs, apply_bc=1) if rhs else None
    g = gpu_assemble(t, xyz, conn, ops, rhs=rhs, k=k, bc=pair)
    b = np.zeros(ndof)
    for op, mat in zip(ops, g["mats"]):
        csr, bo = O.build(t, xyz, conn, em, ndof, lhs=oracle_lhs(op, k), bc_mask=mask, bc_val=val, nthreads=4)
        assert compare_csr(mat, csr, ndof, what="tet fixed point") == 0
        if bc:
            b += bo
    if rhs:
        b += O.build(t, xyz, conn, em, ndof, rhs={"kind": 1, "fn": rhs["fn"], "c": rhs["coef"],
                                                  "apply_bc": rhs["apply_bc"]}, bc_mask=mask, bc_val=val)[1]
    if rhs or bc:
        assert_close(g["b"], b, what="tet fixed point b")


@pytest.mark.parametrize("n", [1, 2, 3, 5])
@pytest.mark.parametrize("t", [O.P1TET, O.P2TET], ids=["p1", "p2"])
def test_sizes(engine, t, n):
    # 5, 40, 135, 625 elements: partial groups of 32 and blocks of 64; n = 1: too large for
    # the series
    xyz, conn, k = problem("tet5", n, 0.15, seed=5, sigma=0.7)
    check(t, xyz, conn, k, [K_OP, M_OP], SIN3)


@pytest.mark.parametrize("scale", [(0.01, 0.01, 0.01), (0.3, 0.2, 0.1), (1.0, 0.3, 0.01), (2e-40, 1e-40, 1e-40)])
@pytest.mark.parametrize("t", [O.P1TET, O.P2TET], ids=["p1", "p2"])
def test_units(engine, t, scale):
    # degrees 7 to 15 of the series, coordinates with units of their own, tiny elements; 3,750
    # elements and 13,230 take the two routes of the P1 load
    for n in (5, 13) if t == O.P1TET else (4,):
        xyz, conn, k = problem("tet6", n, 0.1, seed=8, sigma=1.0)
        if scale[2] == 0.01 and scale[0] == 1.0:
            check_long_double(t, xyz * np.array(scale), conn, k)
        else:
            check(t, xyz * np.array(scale), conn, k, [K_OP], SIN3)


@pytest.mark.parametrize("bc", [False, True], ids=["nobc", "bc"])
@pytest.mark.parametrize("ops", [[K_OP], [M_OP], [{"stiffness": 1, "stiff_coef": 2.0, "mass": 1, "mass_coef": 0.5}],
                                 [K_OP, M_OP], [M_OP, K_OP]], ids=["K", "M", "K+M in one", "K, M", "M, K"])
@pytest.mark.parametrize("t", [O.P1TET, O.P2TET], ids=["p1", "p2"])
def test_operators(engine, t, ops, bc):
    xyz, conn, k = problem("tet6", 4, 0.12, seed=2, sigma=0.5)
    check(t, xyz, conn, k, ops, SIN3, bc=bc)


def test_refused_coefficients(engine):
    xyz, conn, k = problem("tet6", 3, 0.12, seed=2, sigma=0.5)
    k[::5] = 0.0
    k[1::7] *= -1.0
    k[2] = 1e-310
    check(O.P1TET, xyz, conn, k, [K_OP, M_OP])
