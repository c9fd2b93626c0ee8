"""The waits of the persistent CG: a barrier that is never complete ends with PXG_ERR_TIMEOUT and leaves the
context usable; solves of several contexts at a time, beside other work, and beside a batch give what
they give alone."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def system(n, seed):
    """tridiagonal, strictly diagonally dominant"""
    r = np.random.RandomState(seed)
    off = r.uniform(-0.45, 0.45, n - 1)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.r_[2, np.full(n - 2, 3), 2])
    ci = np.concatenate([[0, 1], np.stack([np.arange(n - 2), np.arange(1, n - 1), np.arange(2, n)], 1).reshape(-1),
                         [n - 2, n - 1]]).astype(np.int32)
    v = np.concatenate([[1.0, off[0]], np.stack([off[:-1], np.ones(n - 2), off[1:]], 1).reshape(-1), [off[-1], 1.0]])
    return [torch.from_numpy(a).to(DEV) for a in (rp, ci, v, r.standard_normal(n))]


@pytest.mark.parametrize("n", [100, 90001])
def test_timeout_is_reported(engine, monkeypatch, n):
    from proxpde_gb300 import Context, PxgError

    rp, ci, v, b = system(n, 1)
    x = torch.empty_like(b)
    ctx = Context(0)
    monkeypatch.setenv("PXG_TEST_BARRIER_SHORTFALL", "1")
    with pytest.raises(PxgError) as ei:
        ctx.cg(rp, ci, v, b, x, rtol=1e-10, max_iter=100)
    assert ei.value.status == 4
    monkeypatch.setenv("PXG_TEST_BARRIER_SHORTFALL", "0")
    _, rel = ctx.cg(rp, ci, v, b, x, rtol=1e-10, max_iter=100)
    assert rel <= 1e-10


def test_solves_of_several_threads(engine):
    from proxpde_gb300 import Context

    sizes = [90001, 30011, 90001, 700]
    data = [system(n, 3 + i) for i, n in enumerate(sizes)]
    alone = []
    for rp, ci, v, b in data:
        x = torch.empty_like(b)
        Context(0).cg(rp, ci, v, b, x, rtol=1e-11, max_iter=200)
        alone.append(x)
    torch.cuda.synchronize()
    got, errors = [None] * len(data), []

    def work(i):
        try:
            ctx = Context(0)
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                rp, ci, v, b = data[i]
                for _ in range(8):
                    x = torch.full_like(b, np.nan)
                    big = torch.randn(1 << 22, device=DEV).sort()  # other work on the GPU
                    ctx.cg(rp, ci, v, b, x, rtol=1e-11, max_iter=200, stream=s.cuda_stream)
                got[i] = x
                del big
            s.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(data))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors
    for a, b in zip(alone, got):
        assert torch.equal(a, b)  # reproducible: sums in a fixed order
