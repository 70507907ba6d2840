"""The 2D kernels from the sources to the cut level's expansions and from there
to the points against the oracle, where their tiles
and the rules of their dispatch end: orders on either side of the tiles of
eight powers and of 32 (eps 1e-3 to 1e-15), leaves of a few sources (a warp
each) and of hundreds (a CTA each), leaves cut into several partial blocks,
evaluation at one point, at remainders of sixteen and with derivatives, several
densities, dipoles; and calls on either side of 3000 points, whose trees are
built on the host and on the device.

FP64, other orders of summation than the oracle's: relative l2 <= 1e-12 for
the potential, a digit more per derivative, as for every FP64 route.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOLS = (("pot", 1e-12), ("pottarg", 1e-12), ("gradtarg", 1e-11), ("hesstarg", 1e-10))

CASES = [  # kind, ns, nt, delta, eps, nd, dipoles, pgh
    ("uniform", 4000, 1, 2e-3, 1e-3, 1, 0, 3),
    ("uniform", 4001, 5003, 2e-3, 1e-6, 1, 0, 2),
    ("uniform", 4001, 3001, 2e-3, 1e-6, 2, 1, 1),
    ("uniform", 6007, 2017, 2e-3, 1e-9, 1, 0, 3),
    ("uniform", 6007, 9001, 2e-3, 1e-12, 1, 1, 2),
    ("uniform", 5000, 1777, 2e-3, 1e-15, 1, 0, 3),
    ("cluster", 8009, 3005, 2e-3, 1e-6, 1, 0, 1),
    ("cluster", 8009, 3005, 2e-3, 1e-12, 2, 0, 2),
    ("uniform", 9001, 2003, 0.1, 1e-6, 2, 0, 2),  # leaves of several partial blocks
    ("uniform", 9001, 2003, 0.1, 1e-9, 1, 1, 1),
    ("uniform", 2048, 513, 0.1, 1e-6, 1, 0, 1),   # a leaf of exactly one block
    ("uniform", 3500, 901, 5e-2, 1e-18, 1, 0, 2),  # node halves beyond 32
    ("cluster", 12007, 4001, 5e-4, 1e-9, 2, 1, 2),  # leaves at several depths
    ("uniform", 2000, 1000, 2e-3, 1e-6, 1, 0, 1),  # 3000 points: host tree
    ("uniform", 2000, 1001, 2e-3, 1e-6, 1, 0, 1),
]


@pytest.mark.parametrize("case", CASES, ids=["_".join(str(v) for v in c) for c in CASES])
def test_form_eval2d_matches_oracle(fgt, oracle, case):
    kind, ns, nt, delta, eps, nd, dip, pgh = case
    rng = np.random.default_rng(ns + nt)
    src, trg = rng.random((ns, 2)), rng.random((nt, 2))
    if kind == "cluster":
        src[: ns // 2] = 0.37 + 5e-3 * rng.random((ns // 2, 2))
    q = rng.standard_normal((ns, nd))
    rn, ds = (rng.standard_normal((ns, 2)), rng.standard_normal((ns, nd))) if dip else (None, None)
    ctx = fgt.Context(0, precision="fp64")
    got = fgt.transform_pgh(2, nd, delta, eps, src, q, trg, 1, pgh, ctx=ctx, ifdipole=dip, rnormal=rn, dipstr=ds)
    ref = oracle.fgt_full(2, nd, delta, eps, src, q, trg, 1, pgh, rn, ds)
    for k, tol in TOLS:
        if got[k] is None:
            continue
        e = oracle.derr(ref[k], got[k])
        print(f"{case}: {k} {e:.2e}")
        assert e <= tol, (k, e)


@pytest.mark.parametrize("eps", [1e-6, 1e-12])
def test_expansions_below_the_cut_2d(fgt, oracle, eps):
    """Formed on request: <= 1e-12 of their largest coefficient."""
    rng = np.random.default_rng(5)
    src = rng.random((8000, 2))
    src[:4000] = 0.37 + 5e-3 * rng.random((4000, 2))
    q = rng.standard_normal((8000, 1))
    plan = fgt.Plan(fgt.Context(0, precision="fp64"), 2, 1, 2e-3, eps, src, None, 1, 0)
    plan.execute_host(src, q)
    inf = plan.info()
    T = fgt.HostTree(2, 2e-3, eps, src, src)
    cut = max(inf["npwlevel"], 0)
    below = [b for b in range(T["nboxes"]) if T["ilevel"][b] > cut]
    pick = sorted(rng.choice(below, size=min(60, len(below)), replace=False).tolist())
    mp, _, has = oracle.expansions(2, 1, 2e-3, eps, src, q, None, 1, 0, pick, inf["nexp"])
    got = [plan.expansion("mp", b) for b in pick]
    plan.close()
    n = 0
    for i, b in enumerate(pick):
        scale = np.abs(mp[i]).max() if has[i] else 0.0
        if scale == 0.0:
            continue
        assert got[i] is not None
        assert np.abs(got[i] - mp[i]).max() <= 1e-12 * scale, b
        n += 1
    assert n > 10
