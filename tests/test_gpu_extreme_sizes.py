"""Elements of extreme size at the origin: lengths times a power of two scale stiffness, mass and (near
zero, where the sine is linear) the sine load by powers of two, down to where they leave the range of
doubles, below which they are zero or subnormal and never large."""
import numpy as np
import pytest

import oracle as O
from helpers import gpu_assemble, problem

pytestmark = pytest.mark.gpu

K_OP = {"stiffness": 2, "stiff_coef": 1.0}
SIN3 = {"kind": 1, "fn": O.FN_SIN3, "coef": 1.0}


def assemble(t, gen, s, mass):
    xyz, conn, k = problem(gen, 3, 0.15, seed=3, sigma=0.5)
    g = gpu_assemble(t, xyz * s, conn, [K_OP, {"mass": 1, "mass_coef": mass}], rhs=SIN3, k=k)
    return [*g["struct_vals"], g["b"]]


@pytest.mark.parametrize("mass", [1.0, 2.0 ** -200], ids=["1", "2^-200"])
@pytest.mark.parametrize("p", [-120, -165, -172, -180, -200, -290])
@pytest.mark.parametrize("t,gen", [(O.P1TET, "tet6"), (O.P2TET, "tet6"), (O.Q1HEX, "hex"), (O.Q2HEX, "hex")],
                         ids=["p1", "p2", "q1", "q2"])
def test_small(engine, t, gen, p, mass):
    base = -100
    for v, v0, power, c in zip(assemble(t, gen, 2.0 ** p, mass), assemble(t, gen, 2.0 ** base, 1.0), (1, 3, 6),
                               (1.0, mass, 1.0)):
        # the reference's exponents in two steps, as they leave the range together with the result
        e = power * (p - base) + int(np.log2(c))
        ref = np.ldexp(np.ldexp(v0, e // 2), e - e // 2)
        # powers of two scale every rounding alike, but for the sine's cubic term ((pi s)^2 / 6 < 2^-200) and,
        # below 2^-900, the cofactor products of elements that FP64 takes; sums of up to 24 elements in any
        # order: 48 half ulps of the largest entry; below the normal range anything up to it
        tol = 48 * 2.0 ** -53 * np.abs(ref).max() + 2.0 ** -1022 * 24
        assert np.isfinite(v).all()
        assert np.abs(v - ref).max() <= tol
