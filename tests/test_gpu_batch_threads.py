"""Batches whose CTAs keep different amounts of shared memory, solved in turn
and by several threads at once, each on a context and a stream of its own."""
import threading

import pytest
import torch

from arcanefem_gb300 import batch as B
from arcanefem_gb300 import fem

pytestmark = pytest.mark.gpu


def options(k):
    """Loose enough for short solves, and never the same twice: each solve enqueues its launch anew."""
    return fem.solver_options(rtol=1e-2 * (1.0 + 1e-6 * k), inner_rtol=0.1, max_iter=20000)


def make(size):
    ctx = fem.Context(torch.cuda.Stream())
    with torch.cuda.stream(ctx.stream):
        bt = B.Batch(ctx, [size], seed=1, jitter=0.2)
    bt.set_config(512, 1, 3.5)
    return ctx, bt


def test_batches_of_different_shared_memory_in_turn():
    made = [make(200), make(20)]
    torch.cuda.synchronize()
    want = []
    for _, bt in made:
        assert bt.solve(options(0))[0][0].status == 0
        want.append(bt.x[0].clone())
    for _ in range(3):                       # the kept launches, after another batch's
        for (_, bt), x in zip(made, want):
            bt.x[0].zero_()
            torch.cuda.synchronize()
            assert bt.solve(options(0))[0][0].status == 0
            assert torch.equal(bt.x[0], x)


def test_batches_of_different_shared_memory_at_once():
    made = [make(200), make(20), make(8), make(120)]
    torch.cuda.synchronize()
    failed = []

    def work(bt):
        try:
            for k in range(400):
                if bt.solve(options(k))[0][0].status:
                    raise AssertionError("not converged")
        except Exception as e:               # noqa: BLE001 - reported below
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(bt,)) for _, bt in made]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[0]
