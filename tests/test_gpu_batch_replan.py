"""A batch call's plan is kept for the next call with the same problems and made again for others: batches
together, alone, in the other order, and set again with other problem boundaries, in turn."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [False, True])
def test_batches_in_turn(engine, use_graph):
    from proxpde_gb300 import batch

    probs = batch.make_problems(n_hex=7, n_tet=5, nmin=2, nmax=9, seed=8)
    A, B = batch.Batch(probs[:7]), batch.Batch(probs[7:])
    alone = {}
    for k, b in (("A", A), ("B", B)):
        fresh = batch.Batch(probs[:7] if k == "A" else probs[7:])
        loss, _ = batch.batch_adjoint([fresh], rtol=1e-12, use_graph=False)
        alone[k] = (np.array(loss), fresh.grad.clone())
    for order in ("AB", "AB", "A", "BA", "B", "AB", "A", "A", "BA"):
        pair = [{"A": A, "B": B}[k] for k in order]
        for b in pair:
            b.grad.fill_(float("nan"))
        losses, _ = batch.batch_adjoint(pair, rtol=1e-12, use_graph=use_graph)
        at = 0
        for k, b in zip(order, pair):
            loss, grad = alone[k]
            # both solve to a residual of 1e-12, the matrices' condition is below 1e4
            assert np.abs(np.array(losses[at:at + len(loss)]) - loss).max() <= 1e-8 * np.abs(loss).max()
            assert float((b.grad - grad).norm()) <= 1e-8 * float(grad.norm())
            at += len(loss)


def test_other_boundaries(engine):
    """The same union mesh as two problems, then as one of both: the loss is the sum, the gradient the same."""
    from proxpde_gb300 import batch

    b = batch.Batch(batch.make_problems(n_hex=2, n_tet=0, nmin=3, nmax=5, seed=2))
    two, _ = batch.batch_adjoint([b], rtol=1e-12, use_graph=True)
    grad = b.grad.clone()
    off, n = b.elem_off, b.nprob

    def bounds(o):
        o = np.ascontiguousarray(o, dtype=np.int64)
        b.ctx._check(b.ctx.L.pxg_batch_set(b.ctx.h, o.ctypes.data_as(C.POINTER(C.c_int64)), o.size - 1), "batch_set")
        b.nprob = o.size - 1

    bounds([off[0], off[-1]])
    one, _ = batch.batch_adjoint([b], rtol=1e-12, use_graph=True)
    assert abs(one[0] - sum(two)) <= 1e-8 * abs(one[0])
    assert float((b.grad - grad).norm()) <= 1e-8 * float(grad.norm())
    bounds(off)
    assert b.nprob == n
    again, _ = batch.batch_adjoint([b], rtol=1e-12, use_graph=True)
    assert np.abs(np.array(again) - np.array(two)).max() <= 1e-8 * max(two)


def test_other_conditions(engine):
    """The captured launches follow the context: other Dirichlet conditions between two calls."""
    from proxpde_gb300 import batch

    probs = batch.make_problems(n_hex=3, n_tet=0, nmin=3, nmax=5, seed=6)

    def conditions(b, every, diag):
        ids = np.arange(0, b.ndof, every, dtype=np.uint32)
        b.ctx.set_bc(ids, np.linspace(0.0, 1.0, ids.size), diag)

    b = batch.Batch(probs)
    for every, diag in ((5, 1.0), (5, 3.0), (7, 1.0), (2, 0.5)):
        conditions(b, every, diag)
        got, _ = batch.batch_adjoint([b], rtol=1e-12, use_graph=True)
        fresh = batch.Batch(probs)
        conditions(fresh, every, diag)
        want, _ = batch.batch_adjoint([fresh], rtol=1e-12, use_graph=False)
        assert np.abs(np.array(got) - np.array(want)).max() <= 1e-8 * np.abs(want).max()
        assert float((b.grad - fresh.grad).norm()) <= 1e-8 * float(fresh.grad.norm())
