"""A 3D leaf of many partial Hermite blocks (240 sources each in a plan of this
size, 78 with dipoles): up to 32 are added where they are read, more by
k_sum_blocks first.  Against the oracle at the edge and beyond, the expansion
of the leaf's box too (FP64, the same sums in another order: relative l2 and
largest coefficient <= 1e-12, as for every FP64 route)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-3, 1e-6])
@pytest.mark.parametrize("blocks,more,nd,dip", [(32, 0, 1, 0), (32, -60, 1, 0), (32, 1, 1, 0), (41, 7, 2, 0), (32, 0, 1, 1), (33, 0, 1, 1)])
def test_partial_blocks(fgt, oracle, blocks, more, nd, dip, eps):
    import torch
    from torch.profiler import ProfilerActivity, profile
    m = blocks * (78 if dip else 240) + more
    rng = np.random.default_rng(m)
    src = rng.random((m + 400, 3))
    src[:m] = 0.37 + 1e-7 * src[:m]
    q = rng.standard_normal((m + 400, nd))
    rn, ds = (rng.standard_normal((m + 400, 3)), rng.standard_normal((m + 400, nd))) if dip else (None, None)
    ctx = fgt.Context(0, precision="fp64")
    plan = fgt.Plan(ctx, 3, nd, 2e-2, eps, src, None, 1, 0, 1, dip)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:  # the first kernels may not be recorded
        plan.execute_host_full(q, rn, ds)
        got = plan.execute_host_full(q, rn, ds)["pot"]
        torch.cuda.synchronize()
    summed = any("k_sum_blocks" in e.name for e in prof.events())
    T = fgt.HostTree(3, 2e-2, eps, src, src[:0])
    count = T["isrcse"].reshape(-1, 2)[:, 1] - T["isrcse"].reshape(-1, 2)[:, 0] + 1
    box = int(np.flatnonzero((T["nchild"] == 0) & (count >= m))[0])
    mp, _, _ = oracle.expansions(3, nd, 2e-2, eps, src, q, None, 1, 0, [box], plan.info()["nexp"]) if not dip else (None,) * 3
    exp = plan.expansion("mp", box)
    plan.close()
    ref = oracle.fgt_full(3, nd, 2e-2, eps, src, q, None, 1, 0, rn, ds)["pot"]
    # the leaf holds a few of the other points too
    assert summed == (count[box] > 32 * (78 if dip else 240))
    assert oracle.derr(ref, got) <= 1e-12
    if mp is not None:
        assert np.abs(exp - mp[0]).max() <= 1e-12 * np.abs(mp[0]).max()
