"""The fixed-point Q1 kernel (csrc/pxg_q1fx.cu) where it can go wrong: element counts
around its 32-element blocks, units and shifts of every kind (meshes near the origin, tiny,
rotated, flat along an axis or a diagonal, degenerate spots), loads on either side of the
sine series' range, the other loads, coefficients it refuses, and operator mixes, against
the oracle under the entrywise rule of helpers.py."""
import numpy as np
import pytest

import oracle as O
from helpers import assert_close, compare_csr, gpu_assemble, oracle_lhs, problem

pytestmark = pytest.mark.gpu

K_OP = {"stiffness": 2, "stiff_coef": 1.0}
M_OP = {"mass": 1, "mass_coef": 1.0}
SIN3 = {"kind": 1, "fn": O.FN_SIN3, "coef": 1.0}


def rotation(seed):
    q, r = np.linalg.qr(np.random.RandomState(seed).standard_normal((3, 3)))
    return q * np.sign(np.diag(r))


def mesh(name, n):
    xyz, conn, k = problem("hex", n, 0.2, seed=11, sigma=1.0)
    if name == "corner":  # every load value is tiny
        xyz = xyz * 1e-3
    elif name == "tiny":
        xyz = xyz * 2.0 ** -120
    elif name == "rotated":
        xyz = xyz @ rotation(3).T * 0.4
    elif name == "flat":
        xyz = xyz * np.array([1.0, 0.5, 1e-3])
    elif name == "flat rotated":  # the oracle's J loses |x| / thickness: keep it mild
        xyz = xyz * np.array([1.0, 1.0, 0.05]) @ rotation(4).T
    elif name == "graded":  # elements of very different shapes in one block
        xyz = xyz ** np.array([1.0, 2.0, 4.0])
    elif name == "wedges":  # collapsed edges: the determinant vanishes towards one side
        z = xyz[:, 2].copy()
        xyz[:, 0] = xyz[:, 0] * (0.02 + z)
    return xyz, conn, k


def long_double(xyz, conn, k, em, ndof):
    """K(k), M as dense matrices and the sine load in numpy's long double (64-bit or longer
    significand): the oracle's J and Gram determinant lose about the square of an element's
    aspect ratio, more than the tolerance, on meshes flatter than 1:100."""
    f = np.longdouble
    g = f(0.5773502691896258)
    bits = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]])
    sg = (2 * bits - 1).astype(f)
    X = xyz[conn.astype(np.int64)].astype(f)
    origin = X.mean(axis=1)
    K, M, b = np.zeros((ndof, ndof), f), np.zeros((ndof, ndof), f), np.zeros(ndof, f)
    for q in range(8):
        xi = sg[q] * g
        l, h = (1 + sg * xi) / 2, f(0.5)
        phi = l.prod(axis=1)
        dphi = h * sg * np.stack([l[:, 1] * l[:, 2], l[:, 0] * l[:, 2], l[:, 0] * l[:, 1]], axis=1)
        J = np.einsum("enr,nd->erd", X - X[:, :1], dphi)
        a, c, d = J[:, :, 0], J[:, :, 1], J[:, :, 2]
        C = np.stack([np.cross(c, d), np.cross(d, a), np.cross(a, c)], axis=1)  # cofactors by direction
        det = np.abs((a * C[:, 0]).sum(axis=1))
        D = np.einsum("nd,edr->enr", dphi, C)
        Ke = np.einsum("enr,emr->enm", D, D) * (k / det)[:, None, None]
        fq = np.sin(f(np.pi) * (origin + np.einsum("erd,d->er", J, xi))).prod(axis=1)
        e = em.astype(np.int64)
        np.add.at(K, (e[:, :, None], e[:, None, :]), Ke)
        np.add.at(M, (e[:, :, None], e[:, None, :]), det[:, None, None] * (phi[:, None] * phi))
        np.add.at(b, e, (det * fq)[:, None] * phi)
    return K, M, b


def check(xyz, conn, k, ops, rhs, field=None, bc=None):
    em, ndof = O.dofmap(O.Q1HEX, xyz.shape[0], conn)
    g = gpu_assemble(O.Q1HEX, xyz, conn, ops, rhs=rhs, k=k, field=field, bc=bc)
    for op, mat in zip(ops, g["mats"]):
        csr, _ = O.build(O.Q1HEX, xyz, conn, em, ndof, lhs=oracle_lhs(op, k), nthreads=4)
        assert compare_csr(mat, csr, ndof, what="q1 fixed point") == 0
    if rhs is not None:
        r = {"kind": rhs["kind"], "fn": rhs.get("fn", 0), "c": rhs["coef"]}
        if field is not None:
            r["field"] = field
        _, b = O.build(O.Q1HEX, xyz, conn, em, ndof, rhs=r)
        assert_close(g["b"], b, what="q1 fixed point b")


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7])
def test_sizes(engine, n):
    # n <= 4: elements too large for the series in part; 1, 8, 27, 64, 125, 343 elements
    xyz, conn, k = mesh("cube", n)
    check(xyz, conn, k, [K_OP, M_OP], SIN3)


@pytest.mark.parametrize("name", ["corner", "tiny", "rotated", "flat", "flat rotated", "graded", "wedges"])
def test_shapes(engine, name):
    xyz, conn, k = mesh(name, 6)
    if name != "flat":
        return check(xyz, conn, k, [K_OP, M_OP], SIN3)
    em, ndof = O.dofmap(O.Q1HEX, xyz.shape[0], conn)
    K, M, b = long_double(xyz, conn, k, em, ndof)
    g = gpu_assemble(O.Q1HEX, xyz, conn, [K_OP, M_OP], rhs=SIN3, k=k)
    for ref, (rp, ci, v) in zip((K, M), g["mats"]):
        rows = np.repeat(np.arange(ndof), np.diff(rp))
        o = (rp, ci, ref[rows, ci].astype(np.float64))
        assert compare_csr((rp, ci, v), o, ndof, what="q1 fixed point flat") == 0
    assert_close(g["b"], b.astype(np.float64), what="q1 fixed point flat b")


@pytest.mark.parametrize("scale", [0.02, 0.3, 1.7])
def test_series_degrees(engine, scale):
    # |pi d| around 0.004, 0.06 and 0.35: degrees 7, 9, 15
    xyz, conn, k = mesh("cube", 6)
    check(xyz * scale, conn, k, [], SIN3)


@pytest.mark.parametrize("rhs", [{"kind": 1, "fn": O.FN_CONST, "coef": -2.5},
                                 {"kind": 1, "fn": O.FN_POISSON_RHS, "coef": 0.5}, {"kind": 2, "coef": 1.5}],
                         ids=["const", "poisson", "projection"])
def test_other_loads(engine, rhs):
    xyz, conn, k = mesh("cube", 5)
    field = None
    if rhs["kind"] == 2:
        _, ndof = O.dofmap(O.Q1HEX, xyz.shape[0], conn)
        field = np.cos(np.arange(ndof))
    check(xyz, conn, k, [K_OP], rhs, field=field)


def test_refused_elements(engine):
    # zero, negative and subnormal coefficients: refused ones among the others of a block
    xyz, conn, k = mesh("cube", 5)
    k[::7] = 0.0
    k[1::5] *= -1.0
    k[3] = 1e-310
    check(xyz, conn, k, [K_OP, M_OP], SIN3)


@pytest.mark.parametrize("ops", [[K_OP], [M_OP], [{"stiffness": 1, "stiff_coef": 2.0, "mass": 2, "mass_coef": 0.5}],
                                 [{"stiffness": 2, "stiff_coef": 1.0, "mass": 1, "mass_coef": 3.0}, K_OP],
                                 [M_OP, {"stiffness": 1, "stiff_coef": 0.25}]],
                         ids=["K", "M", "K+kM", "K+M,K", "M,K"])
def test_operator_mixes(engine, ops):
    xyz, conn, k = mesh("cube", 5)
    check(xyz, conn, k, ops, None)
