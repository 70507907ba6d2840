"""Plans of few points (their tree is built on the host) beside other work of
the program: the caller's arrays and the streams they may touch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stall(stream, seconds=0.3):
    """Work of about that long queued on the stream, and its end."""
    import torch
    end = torch.cuda.Event()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(int(seconds * 1.9e9))
        end.record(stream)
    return end


@pytest.mark.parametrize("delta", [1e-3, 10.0], ids=["tree", "large_delta"])
@pytest.mark.parametrize("tree", [None, "host"])
def test_points_may_change_after_plan_creation(fgt, delta, tree):
    """Pinned point arrays are read before the plan's creation returns, even
    when the context's stream is busy."""
    import torch
    ctx = fgt.Context(0) if tree is None else fgt.Context(0, tree=tree)
    rng = np.random.default_rng(8)
    n = 900
    src, trg, q = rng.random((n, 2)), rng.random((n, 2)), rng.random((n, 1))
    plan = fgt.Plan(ctx, 2, 1, delta, 1e-6, src, trg, 1, 1)
    ref = plan.execute_host(src, q, trg)
    plan.close()
    hs, ht = (torch.from_numpy(a.copy()).pin_memory() for a in (src, trg))
    _stall(torch.cuda.ExternalStream(ctx.stream))
    plan = fgt.Plan(ctx, 2, 1, delta, 1e-6, hs.numpy(), ht.numpy(), 1, 1)
    hs.zero_()
    ht.zero_()
    got = plan.execute_host(src, q, trg)
    plan.close()
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("entry", ["plan", "call"])
@pytest.mark.parametrize("tree", [None, "host"])
def test_no_wait_for_the_default_stream(fgt, entry, tree):
    """A plan, its execute and a drop-in call run beside work on the default
    stream instead of after it."""
    import torch
    ctx = fgt.Context(0) if tree is None else fgt.Context(0, tree=tree)
    rng = np.random.default_rng(9)
    n = 900
    src, q = rng.random((n, 2)), rng.random((n, 1))

    def go():
        if entry == "call":
            return fgt.transform(2, 1, 1e-3, 1e-6, src, q, ctx=ctx)[0]
        plan = fgt.Plan(ctx, 2, 1, 1e-3, 1e-6, src, None, 1, 0)
        pot = plan.execute_host(src, q)[0]
        plan.close()
        return pot

    ref = go()
    end = _stall(torch.cuda.default_stream(), 0.5)
    got = go()
    waited = end.query()
    torch.cuda.synchronize()
    assert np.array_equal(got, ref) and not waited
