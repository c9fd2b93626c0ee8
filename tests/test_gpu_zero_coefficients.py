"""Elements whose coefficient is zero: exact zeros in the matrices, at the price of other elements (the
element kernels once sent each to a slow path of its own)."""
import numpy as np
import pytest

import oracle as O
from helpers import compare_csr, gpu_assemble, oracle_lhs, problem

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

K_OP = {"stiffness": 2, "stiff_coef": 1.0}
M_OP = {"mass": 2, "mass_coef": 2.0}
ELEMENTS = [(O.P1TET, "tet6", 5), (O.P2TET, "tet6", 3), (O.Q1HEX, "hex", 5), (O.Q2HEX, "hex", 3)]


@pytest.mark.parametrize("share", [0.3, 1.0])
@pytest.mark.parametrize("t,gen,n", ELEMENTS, ids=[O.NAMES[e[0]] for e in ELEMENTS])
def test_values(engine, t, gen, n, share):
    xyz, conn, k = problem(gen, n, 0.15, seed=9, sigma=0.5)
    k[np.random.RandomState(0).uniform(size=k.size) < share] = 0.0
    em, ndof = O.dofmap(t, xyz.shape[0], conn)
    for ops in ([K_OP, M_OP], [K_OP], [{"stiffness": 1, "stiff_coef": 0.0, "mass": 1, "mass_coef": 1.0}]):
        g = gpu_assemble(t, xyz, conn, ops, k=k)
        for op, mat, v in zip(ops, g["mats"], g["struct_vals"]):
            csr, _ = O.build(t, xyz, conn, em, ndof, lhs=oracle_lhs(op, k))
            if csr[2].size:
                compare_csr(mat, csr, ndof, what="zero coefficients")
            else:
                assert not v.any()


@pytest.mark.parametrize("t,gen,n", [(O.P1TET, "tet6", 40), (O.P2TET, "tet6", 20), (O.Q1HEX, "hex", 43),
                                     (O.Q2HEX, "hex", 16)], ids=["p1", "p2", "q1", "q2"])
def test_price(engine, t, gen, n):
    from proxpde_gb300 import Context

    xyz, conn, k = problem(gen, n, 0.15, seed=9, sigma=0.5)
    c = Context(0)
    c.set_mesh(t, xyz, conn)
    ndof = c.build_dofmap()
    vals = [torch.empty(c.build_pattern(), dtype=torch.float64, device="cuda:0") for _ in range(2)]

    def best(coef):
        c.set_coef(coef)
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                c.assemble(op0=K_OP, vals0=vals[0], op1=M_OP, vals1=vals[1])
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    zero = np.where(np.random.RandomState(0).uniform(size=k.size) < 0.5, 0.0, k)
    # the same work up to the reductions of zeros; on the slow path 1.1 (P1) to 6 times the time
    assert best(zero) <= 1.08 * best(k)
