"""What a launch reports when a CTA waits for longer than its limit: by priority class the wait is for any
ready task, in the one queue for the slot the CTA has drawn.  The limit is one microsecond here, less
than any instruction takes, so the CTAs that find nothing give up at once and the others finish what is
ready.  Which queue a program takes shows in the message."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def instances(pp, ctx, count):
    hs = []
    for i in range(count):
        h, _ = pp.make_dense_problem(ctx, n=256, leaf=64, seed=i)
        h.upload()
        h.keep_original()
        hs.append(h)
    return hs


def test_nothing_ready_by_class(pp, gctx):
    ctx = pp.Context(device=0, spin_limit=1)
    batch = pp.Batch(ctx, instances(pp, ctx, 64))
    for _ in range(2):
        batch.restore()
        batch.factor()
        with pytest.raises(pp.PPError, match="no task became ready within the time limit") as e:
            batch.sync()
        assert e.value.status == pp.PP_TIMEOUT
    # the device and its other contexts go on
    batch = pp.Batch(gctx, instances(pp, gctx, 64))
    batch.factor()
    batch.sync()


def test_slot_of_the_one_queue(pp, gctx):
    ctx = pp.Context(device=0, spin_limit=1)
    h, = instances(pp, ctx, 1)
    h.factor()
    with pytest.raises(pp.PPError, match="ready-queue slot [0-9]+ never filled") as e:
        h.sync()
    assert e.value.status == pp.PP_TIMEOUT
