"""Stiffness of tetrahedra of strongly different shapes (sheared, thin, with short edges and small faces,
slivers), each an element of its own, against the cofactor formula in numpy's long double.  Small entries
belong to small faces and are held to their own size: |K_ab - ref| <= tol sqrt(K_aa K_bb) for the vertices
1 to 3 (vertex 0's row is minus the sum of the others')."""
import numpy as np
import pytest

import oracle as O
from helpers import gpu_assemble

pytestmark = pytest.mark.gpu

K_OP = {"stiffness": 2, "stiff_coef": 1.0}
M_OP = {"mass": 1, "mass_coef": 1.0}
N = 96  # three warps


def edges(shape, eps, seed):
    """(N, 3, 3): edge vectors of vertices 1..3 from vertex 0"""
    r = np.random.RandomState(seed)
    d = np.zeros((N, 3, 3))
    u = r.uniform(0.5, 1.5, (N, 3, 3))
    d[:, 0, 0], d[:, 1, 1], d[:, 2, 2] = u[:, 0, 0], u[:, 1, 1], u[:, 2, 2]
    if shape == "shear":  # two edges nearly parallel, along an axis
        d[:, 1, 0], d[:, 1, 1] = u[:, 1, 0], eps * u[:, 1, 1]
        d[:, 2, 0], d[:, 2, 1] = u[:, 2, 0] - 1, u[:, 2, 1] - 1
    elif shape == "thin":
        d[:, 2, 2] *= eps
        d[:, 2, :2] = u[:, 2, :2] - 1
    elif shape == "short":
        d = r.uniform(-1, 1, (N, 3, 3))
        d[:, 1] *= eps
    elif shape == "face":
        d = r.uniform(-1, 1, (N, 3, 3))
        d[:, 1] = 0.7 * d[:, 0] + eps * d[:, 1]
    elif shape == "flat":
        d = r.uniform(-1, 1, (N, 3, 3))
        d[:, 2] = 0.3 * d[:, 0] + 0.7 * d[:, 1] + eps * d[:, 2]
    return d


@pytest.mark.parametrize("ops", [[K_OP], [K_OP, M_OP]], ids=["K", "K, M"])
@pytest.mark.parametrize("eps", [1.0, 0.03, 1e-3, 1e-5])
@pytest.mark.parametrize("shape", ["shear", "thin", "short", "face", "flat"])
@pytest.mark.parametrize("t", [O.P1TET, O.P2TET], ids=["p1", "p2"])
def test_shapes(engine, t, shape, eps, ops):
    d = edges(shape, eps, 7)
    xyz = np.concatenate([np.zeros((N, 1, 3)), d], axis=1).reshape(-1, 3)  # vertex 0 at the origin: exact differences
    conn = np.arange(4 * N, dtype=np.uint32).reshape(N, 4)
    k = np.exp(np.random.RandomState(1).standard_normal(N))
    g = gpu_assemble(t, xyz, conn, ops, k=k)
    rp, ci, v = g["mats"][0]
    f = np.longdouble
    D = d.astype(f)
    C = np.stack([np.cross(D[:, 1], D[:, 2]), np.cross(D[:, 2], D[:, 0]), np.cross(D[:, 0], D[:, 1])], axis=1)
    det = np.abs((D[:, 0] * C[:, 0]).sum(axis=1))
    # grad lambda_a . grad lambda_b k |T|; a vertex pair's P2 entry is 3/5 of it on the diagonal, -1/5 beside it
    S = np.einsum("ear,ebr->eab", C, C) * (k / det / 6)[:, None, None]
    W = np.ones((3, 3)) if t == O.P1TET else np.full((3, 3), f(-1) / 5) + (f(3) / 5 + f(1) / 5) * np.eye(3, dtype=f)
    # FP64's own bound: the determinant and the cofactors are sums of products that may cancel; with a
    # dozen roundings each, and 4.1e-15 for the 16 digits of the P2 rule
    a = np.abs(D)
    perm = sum(a[:, 0, p] * a[:, 1, q] * a[:, 2, r] for p in range(3) for q in range(3) for r in range(3)
               if len({p, q, r}) == 3)
    P = np.stack([a[:, 1][:, [1, 2, 0]] * a[:, 2][:, [2, 0, 1]] + a[:, 1][:, [2, 0, 1]] * a[:, 2][:, [1, 2, 0]],
                  a[:, 2][:, [1, 2, 0]] * a[:, 0][:, [2, 0, 1]] + a[:, 2][:, [2, 0, 1]] * a[:, 0][:, [1, 2, 0]],
                  a[:, 0][:, [1, 2, 0]] * a[:, 1][:, [2, 0, 1]] + a[:, 0][:, [2, 0, 1]] * a[:, 1][:, [1, 2, 0]]], axis=1)
    cond = perm / det + 2 * (np.sqrt((P * P).sum(2)) / np.sqrt((C * C).sum(2))).max(axis=1)
    tol = 12 * 2.0 ** -53 * cond + 4.1e-15 * (t == O.P2TET)
    em = g["em"]
    K = np.zeros((N, 3, 3), f)
    for p in range(3):
        for q in range(3):
            row, col = em[:, p + 1].astype(int), em[:, q + 1].astype(int)
            for e in range(N):
                at = np.nonzero(ci[rp[row[e]]:rp[row[e] + 1]] == col[e])[0]
                K[e, p, q] = v[rp[row[e]] + at[0]] if at.size else 0.0  # closeMatrix drops tiny entries
    ref = S * W
    scale = np.sqrt(np.einsum("eaa->ea", S)[:, :, None] * np.einsum("eaa->ea", S)[:, None, :])
    bad = np.abs(K - ref) > tol[:, None, None] * scale + 1e-16
    assert not bad.any(), f"{bad.sum()} of {bad.size}, worst {float((np.abs(K - ref) / (tol[:, None, None] * scale)).max()):.3g}"
