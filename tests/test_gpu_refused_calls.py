"""Calls that are refused for a value that is not finite, at sizes on either
side of the smallest tree built on the device: the same status, and the
drop-in call's outputs are zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", ["charge", "source", "target", "dipole"])
@pytest.mark.parametrize("n", [1, 500, 5000])
@pytest.mark.parametrize("tree", [None, "host"])
def test_refused_call_zeroes_its_outputs(fgt, bad, n, tree):
    rng = np.random.default_rng(n)
    src, trg, q = rng.random((n, 2)), rng.random((n, 2)), rng.random((n, 1))
    rn, ds = rng.random((n, 2)), rng.random((n, 1))
    {"charge": q, "source": src, "target": trg, "dipole": ds}[bad][n // 2, 0] = np.nan
    ctx = fgt.Context(0) if tree is None else fgt.Context(0, tree=tree)
    out = {k: np.full(s, 7.0) for k, s in (("pot", (n, 1)), ("grad", (n, 2, 1)), ("pottarg", (n, 1)))}
    with pytest.raises(fgt.FGTError) as e:
        fgt.transform_pgh(2, 1, 1e-3, 1e-6, src, q, trg, 2, 1, ctx, 1, 1, rn, ds, out)
    assert e.value.status == 1
    for k, v in out.items():
        assert np.all(v == 0.0), k


def test_no_sources(fgt):
    """Without sources the fields are zero, whatever the targets hold."""
    trg = np.full((10, 2), np.nan)
    ctx = fgt.Context(0)
    _, pt = fgt.transform(2, 1, 1e-3, 1e-6, np.zeros((0, 2)), np.zeros((0, 1)), trg, 0, 1, ctx=ctx)
    assert np.all(pt == 0.0)


def _stalled(ctx, seconds=0.3):
    """Work of about that long queued on the context's stream, and its end."""
    import torch
    s = torch.cuda.ExternalStream(ctx.stream)
    end = torch.cuda.Event()
    with torch.cuda.stream(s):
        torch.cuda._sleep(int(seconds * 1.9e9))
        end.record(s)
    return end


def test_refused_call_leaves_no_copy_behind(fgt):
    """A one-shot call that is refused for its strengths returns when nothing
    reads the caller's (pinned) arrays any more."""
    import torch
    ctx = fgt.Context(0)
    rng = np.random.default_rng(3)
    pin = [torch.from_numpy(a).pin_memory() for a in (rng.random((500, 2)), rng.random((500, 1)))]
    src, q = (a.numpy() for a in pin)
    fgt.transform(2, 1, 1e-3, 1e-6, src, q, ctx=ctx)
    q[499] = np.inf
    end = _stalled(ctx)
    with pytest.raises(fgt.FGTError) as e:
        fgt.transform(2, 1, 1e-3, 1e-6, src, q, ctx=ctx)
    done = end.query()  # the uploads follow it
    torch.cuda.synchronize()
    assert e.value.status == 1 and done


@pytest.mark.parametrize("bad", ["charge", "rnormal", "dipstr"])
def test_refused_execute_copies_nothing(fgt, bad):
    """Strengths that are looked at on the host are refused before any copy of
    them is queued."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    ctx = fgt.Context(0)
    rng = np.random.default_rng(4)
    n = 500
    plan = fgt.Plan(ctx, 2, 1, 1e-3, 1e-6, rng.random((n, 2)), None, 1, 0, 1, 1)
    a = dict(charge=rng.random((n, 1)), rnormal=rng.random((n, 2)), dipstr=rng.random((n, 1)))
    pot = np.zeros((n, 1))

    def run():
        p = lambda x: fgt._p(x)
        return fgt.lib().fgt_plan_execute_host_full(plan._h, p(a["charge"]), p(a["rnormal"]), p(a["dipstr"]), p(pot),
                                                    None, None, None, None, None)

    assert run() == 0
    a[bad][0, 0] = np.nan
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        st = run()
        torch.cuda.synchronize()
    copies = [e.name for e in prof.events() if "HtoD" in e.name]
    plan.close()
    assert st == 1 and not copies, copies


def test_refused_points_leave_no_upload_behind(fgt):
    """The strengths of a one-shot call go up beside the tree build: a call
    that is refused for its points returns when that upload has ended."""
    import time

    import torch
    rng = np.random.default_rng(6)
    ns, nd = 200000, 256
    q = torch.zeros(ns, nd, dtype=torch.float64).pin_memory().numpy()  # 410 MB, about 8 ms
    src = rng.random((ns, 2))
    src[7, 1] = np.nan
    ctx = fgt.Context(0)
    after = []
    for _ in range(3):
        with pytest.raises(fgt.FGTError):
            fgt.transform_pgh(2, nd, 1e-3, 1e-6, src, q, src[:1], 0, 1, ctx)
        t0 = time.perf_counter()
        torch.cuda.synchronize()
        after.append(time.perf_counter() - t0)
    assert min(after) < 1e-3, after
