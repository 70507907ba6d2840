"""The SM budget and the yielding grids: they size the launches of the
transforms between the leaves and the cut level and change no result."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNELS = {2: ("k_up2d_x", "k_down2d_x"), 3: ("k_up_z", "k_down_xy")}


def _grids(prof, path):
    """CTAs of the largest launch of every kernel."""
    prof.export_chrome_trace(str(path))
    out = {}
    for e in json.load(open(path))["traceEvents"]:
        if e.get("cat") == "kernel":
            g = e["args"]["grid"]
            out[e["name"]] = max(out.get(e["name"], 0), g[0] * g[1] * g[2])
    return out


@pytest.mark.parametrize("dim,n,delta,eps", [(2, 300000, 1e-5, 1e-9), (2, 2000000, 1e-5, 1e-6), (3, 100000, 2e-2, 1e-9)])
def test_grid_switches(fgt, tmp_path, dim, n, delta, eps):
    import torch
    from torch.profiler import ProfilerActivity, profile
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(dim)
    src, q = rng.random((n, dim)), rng.standard_normal((n, 1))
    pots, grids = {}, {}
    for name, budget, on in (("all", 0, False), ("few", 4, False), ("yield", 4, True)):
        ctx = fgt.Context(0, precision="fp64")
        ctx.set_sm_budget(budget)
        ctx.set_grid_yield(on)
        plan = fgt.Plan(ctx, dim, 1, delta, eps, src, None, 1, 0)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:  # the first kernels may not be recorded
            plan.execute_host(src, q)
            pots[name] = plan.execute_host(src, q)[0]
        grids[name] = _grids(prof, tmp_path / f"{name}.json")
        plan.close()
    assert np.array_equal(pots["all"], pots["few"]) and np.array_equal(pots["all"], pots["yield"])
    for k in KERNELS[dim]:
        a, f, y = (max(v for m, v in grids[g].items() if k in m) for g in ("all", "few", "yield"))
        print(k, a, f, y)
        assert f < a, (k, f, a)
        assert y >= a, (k, a, y)
        if dim == 2:
            assert a <= 16 * sms and f <= 16 * 4, (k, a, f)
        if n == 2000000:  # more work than the default grid takes at once
            assert a == 16 * sms < y, (k, a, y)
