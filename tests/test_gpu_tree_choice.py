"""Where a plan's tree is built: the context's choice at any size; without a
choice the device above 3000 points (targets that are the sources count once,
targets that only begin at the same address do not)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RNG = np.random.default_rng(12)
BIG = RNG.random((100000, 2))
SMALL = RNG.random((1500, 2))


@pytest.mark.parametrize("tree,src,trg,device", [
    ("device", SMALL[:500], None, True),
    ("device", SMALL, SMALL, True),
    ("host", BIG[:5000], None, False),
    (None, BIG[:3000], None, False),
    (None, BIG[:3001], None, True),
    (None, BIG[:3000], BIG[:3000], False),
    (None, SMALL, BIG[:1500], False),
    (None, SMALL, BIG[:1501], True),
    (None, BIG[:1000], BIG, True),
    ("auto", SMALL, None, False),
])
def test_tree_choice(fgt, tree, src, trg, device):
    import torch
    from torch.profiler import ProfilerActivity, profile
    ctx = fgt.Context(0) if tree is None else fgt.Context(0, tree=tree)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        plan = fgt.Plan(ctx, 2, 1, 1e-3, 1e-6, src, trg, 1, 0 if trg is None else 1)
        torch.cuda.synchronize()
    plan.close()
    # the device build reads counts and boxes back, the host build nothing
    names = {e.name for e in prof.events()}
    assert any("DtoH" in n for n in names) == device, names
