"""Dirichlet conditions on some of a call's parts only: stiffness and mass in two operators and a load,
each with or without the condensation, for every kind of load and both scatters, against the oracle
under the rule of helpers.py."""
import itertools

import numpy as np
import pytest

import oracle as O
from helpers import assert_close, compare_csr, gpu_assemble, oracle_lhs, problem

pytestmark = pytest.mark.gpu

LOADS = {
    "sin3": {"kind": 1, "fn": O.FN_SIN3, "coef": 1.0},
    "const": {"kind": 1, "fn": O.FN_CONST, "coef": -2.0},
    "poisson": {"kind": 1, "fn": O.FN_POISSON_RHS, "coef": 0.5},
    "projection": {"kind": 2, "coef": 1.5},
    "values": {"kind": 3, "coef": 0.75},
}
ELEMENTS = [(O.P1TET, "tet6", 4), (O.P2TET, "tet6", 3), (O.Q1HEX, "hex", 4), (O.Q2HEX, "hex", 3)]


# 384 and 13,824 P1 tetrahedra take the two routes of their sine load
@pytest.mark.parametrize("scatter", [0, 1], ids=["reduce", "colour"])
@pytest.mark.parametrize("load", LOADS)
@pytest.mark.parametrize("t,gen,n", ELEMENTS + [(O.P1TET, "tet6", 14)],
                         ids=[O.NAMES[e[0]] for e in ELEMENTS] + ["p1tet large"])
def test_each_part_its_own_conditions(engine, t, gen, n, load, scatter):
    xyz, conn, k = problem(gen, n, 0.15, seed=17, sigma=0.5)
    em, ndof = O.dofmap(t, xyz.shape[0], conn)
    x = O.dof_coords(t, xyz, conn, em, ndof)
    mask = O.plane_bc_mask(x, [("x", 0.0)])
    val = np.where(mask, 0.5 + x[:, 1], 0.0)
    ids = np.nonzero(mask)[0].astype(np.uint32)
    rhs, field = dict(LOADS[load]), None
    if rhs["kind"] == 2:
        field = np.cos(np.arange(ndof))
    elif rhs["kind"] == 3:
        p = O.qpoints(t, xyz, conn).reshape(-1, 3)
        field = np.exp(p[:, 0]) * np.cos(2.0 * p[:, 1])
    for bk, bm, br in itertools.product((0, 1), repeat=3):
        ops = [{"stiffness": 2, "stiff_coef": 1.0, "apply_bc": bk}, {"mass": 1, "mass_coef": 3.0, "apply_bc": bm}]
        rhs["apply_bc"] = br
        g = gpu_assemble(t, xyz, conn, ops, rhs=rhs, k=k, bc=(ids, val[ids]), field=field, scatter=scatter)
        b = np.zeros(ndof)
        for op, mat in zip(ops, g["mats"]):
            csr, b = O.build(t, xyz, conn, em, ndof, lhs=oracle_lhs(op, k), bc_mask=mask, bc_val=val, b=b)
            compare_csr(mat, csr, ndof, what="own conditions")
        r = {"kind": rhs["kind"], "fn": rhs.get("fn", 0), "c": rhs["coef"], "apply_bc": br}
        if field is not None:
            r["field"] = field
        _, b = O.build(t, xyz, conn, em, ndof, rhs=r, bc_mask=mask, bc_val=val, b=b)
        assert_close(g["b"], b, what="own conditions b")
