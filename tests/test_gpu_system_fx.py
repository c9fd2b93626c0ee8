"""The component blocks of one vector space: 64-bit fixed point against the FP64 path, which elements
outside the fixed-point range take.  Lengths times a power of two scale the stiffness exactly, so the
same mesh at both scales compares the two."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _assemble(et, n, scale, dim, ops, squeeze):
    from proxpde_gb300 import _lib as L
    from proxpde_gb300 import meshgen

    xyz, conn = (meshgen.cube_hex if et in (L.Q1HEX, L.Q2HEX) else meshgen.cube_tet6)(n)
    lat = np.rint(xyz * n)
    inner = ((lat > 0) & (lat < n)).all(1)
    noise = np.random.RandomState(n).uniform(-0.15 / n, 0.15 / n, xyz.shape)
    xyz = (xyz + np.where(inner[:, None], noise, 0.0)) * np.array([1.0, 1.0, squeeze])
    c = L.Context(0)
    c.set_mesh(et, np.ascontiguousarray(xyz * scale), conn.astype(np.uint32))
    c.build_dofmap()
    S = L.System([c], [dim], qr_types=[et])
    vals = torch.empty(S.nnz, dtype=torch.float64, device="cuda:0")
    b = torch.empty(S.ntot, dtype=torch.float64, device="cuda:0")
    S.assemble(0, 0, ops, vals, b)
    return vals.cpu().numpy()


@pytest.mark.parametrize("etype", ["P1TET", "P2TET", "Q1HEX", "Q2HEX"])
@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("squeeze", [1.0, 0.01])
def test_fixed_point_blocks(etype, dim, squeeze):
    from proxpde_gb300 import _lib as L

    et = getattr(L, etype)
    ops = [(L.OP_TENSOR_STIFFNESS, 0.1), (L.OP_STIFFNESS, 1.0)]
    fixed = _assemble(et, 3, 1.0, dim, ops, squeeze)
    # weighted gradients below 2^-322 are not in the fixed-point range
    s = 2.0 ** -180
    plain = _assemble(et, 3, s, dim, ops, squeeze) / s
    # geometry rounds alike at both scales; an entry is at most 27 terms (27 additions and two products
    # each) from up to 24 elements, whose magnitudes sum to at most the geometric mean of two diagonal
    # entries, with the stiffness' three components counted once more: (27 + 2 + 24) 2^-53 each side
    tol = 2 * 2 * 53 * 2.0 ** -53 * np.abs(plain).max()
    assert np.isfinite(fixed).all()
    assert np.abs(fixed - plain).max() <= tol
