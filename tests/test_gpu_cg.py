"""The device CG (pxg_cg) on matrices whose rows and sizes meet the edges of its tiles: residual of the
solution against a dense FP64 product."""
import functools

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

RTOL = 1e-10


@functools.lru_cache(maxsize=1)
def _matrix(n, half, seed, ragged):
    """Symmetric, strictly diagonally dominant (condition number at most 3) banded CSR; every row's
    band shortened at random where ragged."""
    r = np.random.RandomState(seed)
    i = np.arange(n)
    reach = r.randint(0, half + 1, n) if ragged else np.full(n, half)
    rows, cols, vals = [i], [i], [np.ones(n)]
    for d in range(1, half + 1):
        k = i[(reach >= d) & (i + d < n)]
        v = r.uniform(-1, 1, len(k)) / (4.0 * half)
        rows += [k, k + d]
        cols += [k + d, k]
        vals += [v, v]
    rows, cols, vals = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    order = np.lexsort((cols, rows))
    rows, cols, vals = rows[order], cols[order], vals[order]
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return rp, cols.astype(np.int32), vals.astype(np.float64)


def _mul(rp, ci, v, x):
    return np.add.reduceat(np.append(v * x[ci], 0.0), rp[:-1])


# rows per block under and over a warp's and the block's tiles, one block and all; rows of one entry,
# of 27, of more than a tile's buffer (28 per lane row), and of more than it holds for four rows
@pytest.mark.parametrize("n", [1, 31, 33, 129, 4097, 20011, 90001])
@pytest.mark.parametrize("half,ragged", [(0, False), (1, False), (13, False), (13, True), (14, True), (120, True)])
@pytest.mark.parametrize("offset", [0, 1])
def test_cg_residual(n, half, ragged, offset):
    from proxpde_gb300._lib import Context

    rp, ci, v = _matrix(n, half, n + half, ragged)
    b = np.random.RandomState(n).standard_normal(n)
    dev = "cuda:0"
    # an offset of one entry leaves the 16-byte boundary that the copies into shared memory need
    cd = torch.empty(len(ci) + 4, dtype=torch.int32, device=dev)[offset:offset + len(ci)]
    vd = torch.empty(len(v) + 4, dtype=torch.float64, device=dev)[offset:offset + len(v)]
    cd.copy_(torch.from_numpy(ci))
    vd.copy_(torch.from_numpy(v))
    x = torch.full((n,), np.nan, dtype=torch.float64, device=dev)
    it, rel = Context(0).cg(torch.from_numpy(rp).to(dev), cd, vd, torch.from_numpy(b).to(dev), x, rtol=RTOL,
                            max_iter=200)
    r = b - _mul(rp, ci, v, x.cpu().numpy())
    # the recurrence's residual is under RTOL; it and the true one differ by the rounding of `it` updates
    # of numbers of the right hand side's size, each within (row length + 4) half ulps
    drift = max(it, 1) * (2 * half + 5) * 2.0 ** -52
    assert rel <= RTOL
    assert np.linalg.norm(r) <= (RTOL + drift) * np.linalg.norm(b)


def test_cg_ends():
    from proxpde_gb300._lib import Context, PxgError

    rp, ci, v = _matrix(3000, 13, 5, False)
    dev = "cuda:0"
    a = [torch.from_numpy(t).to(dev) for t in (rp, ci, v)]
    b = torch.ones(3000, dtype=torch.float64, device=dev)
    x = torch.empty_like(b)
    ctx = Context(0)
    it, rel = ctx.cg(*a, torch.zeros_like(b), x, rtol=RTOL, max_iter=10)
    assert it == 0 and rel == 0.0 and not x.any()
    with pytest.raises(PxgError):
        ctx.cg(*a, b, x, rtol=1e-15, max_iter=2)
    first = None
    for _ in range(3):  # reproducible, also after a failed solve
        ctx.cg(*a, b, x, rtol=RTOL, max_iter=100)
        first = x.clone() if first is None else first
        assert torch.equal(first, x)
