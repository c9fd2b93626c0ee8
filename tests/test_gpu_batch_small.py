"""Batches of many small problems, which single warps solve beside the groups of blocks of the larger ones,
against the same problems in batches of few, which blocks solve."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


# 8 to 64 rows a small problem (one to two rows a lane); none, some and many larger ones beside them
@pytest.mark.parametrize("n_hex,n_tet,nmin,nmax", [(400, 0, 1, 3), (0, 700, 1, 2), (500, 400, 1, 5), (350, 300, 3, 8)])
@pytest.mark.parametrize("use_graph", [False, True])
def test_small_problems(engine, n_hex, n_tet, nmin, nmax, use_graph):
    from proxpde_gb300 import batch

    probs = batch.make_problems(n_hex=n_hex, n_tet=n_tet, nmin=nmin, nmax=nmax, seed=3)
    r = np.random.RandomState(1)
    for p in probs:  # conditions on one side, so that every cube has free nodes
        p["bc_nodes"] = np.nonzero(p["xyz"][:, 0] == 0.0)[0]
    B = [batch.Batch(p) for p in (probs[:n_hex], probs[n_hex:]) if p]
    first = None
    for _ in range(2):
        losses, _ = batch.batch_adjoint(B, rtol=1e-12, use_graph=use_graph)
        first = losses if first is None else first
    # a problem's sums are in a fixed order whoever solves it; the assembly's reductions are not
    assert np.abs(first - losses).max() <= 1e-8 * np.abs(losses).max()
    grads = [b.grad_of(p).clone() for b in B for p in range(b.nprob)]
    for q in r.choice(len(probs), 24, replace=False):
        one = batch.Batch([probs[q]])
        loss, _ = batch.batch_adjoint([one], rtol=1e-12, use_graph=False)
        # residual 1e-12 on both sides, condition of the Jacobi-scaled matrices below 1e4
        assert abs(loss[0] - losses[q]) <= 1e-8 * abs(loss[0])
        assert float((one.grad - grads[q]).norm()) <= 1e-8 * float(one.grad.norm())


def test_limits_of_iterations(engine):
    from proxpde_gb300 import PxgError, batch

    probs = batch.make_problems(n_hex=400, n_tet=0, nmin=2, nmax=3, seed=3)
    for p in probs:
        p["bc_nodes"] = np.nonzero(p["xyz"][:, 0] == 0.0)[0]
    b = batch.Batch(probs)
    with pytest.raises(PxgError) as ei:
        batch.batch_adjoint([b], rtol=1e-12, max_iter=2, use_graph=False)
    assert ei.value.status == 5
    losses, it = batch.batch_adjoint([b], rtol=1e-12, use_graph=False)
    assert 2 < it < 65 and np.isfinite(losses).all()
