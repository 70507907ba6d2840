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
