"""The 3D transforms between the leaves and the cut level (fgt_sep3d.cu)
against the oracle, where their tiles end: orders and node counts around the
tiles of eight (eps from 1e-3 to 1e-13), leaves at several depths under one
cut-level box, leaves of more sources than one partial block, a root box at or
above the cut level, several densities, dipoles; and the expansions below the
cut level, formed on request.

FP64, the same routes and orders, other orders of summation: relative l2
<= 1e-12 (expansions: of their largest coefficient), as for every FP64 route.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _points(kind, n, rng):
    x = rng.random((n, 3))
    if kind == "cluster":  # leaves at every depth; one with several partial blocks
        m = n // 2
        x[:m] = 0.37 + 2e-4 * rng.random((m, 3))
        x[m:m + n // 4] = 0.6 + 0.05 * rng.standard_normal((n // 4, 3))
    return x


CASES = [  # kind, n, delta, eps, nd, dipoles
    ("uniform", 5000, 1e-2, 1e-3, 1, 0),
    ("uniform", 6001, 2e-2, 1e-6, 2, 0),
    ("uniform", 2003, 5e-2, 1e-12, 1, 0),
    ("uniform", 1501, 5e-2, 1e-13, 2, 0),
    ("cluster", 20011, 1e-2, 1e-3, 1, 0),
    ("cluster", 20011, 1e-2, 1e-6, 1, 0),
    ("cluster", 9001, 2e-2, 1e-9, 1, 1),
    ("cluster", 2503, 5e-2, 1e-12, 1, 0),
    ("uniform", 3000, 0.5, 1e-6, 1, 0),   # the root box is at or above the cut
    ("uniform", 3000, 0.15, 1e-6, 1, 1),
    ("uniform", 3000, 0.3, 1e-12, 1, 0),
]


@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}_{c[3]:g}_{c[2]:g}" for c in CASES])
def test_sep3d_matches_oracle(fgt, oracle, case):
    kind, n, delta, eps, nd, dip = case
    rng = np.random.default_rng(n)
    src, trg = _points(kind, n, rng), _points(kind, n // 3, rng)
    q = rng.standard_normal((n, nd))
    rn, ds = (rng.standard_normal((n, 3)), rng.standard_normal((n, nd))) if dip else (None, None)
    ctx = fgt.Context(0, precision="fp64")
    got = fgt.transform_pgh(3, nd, delta, eps, src, q, trg, 1, 1, ctx=ctx, ifdipole=dip, rnormal=rn, dipstr=ds)
    ref = oracle.fgt_full(3, nd, delta, eps, src, q, trg, 1, 1, rn, ds)
    for k in ("pot", "pottarg"):
        e = oracle.derr(ref[k], got[k])
        print(f"{case}: {k} {e:.2e}")
        assert e <= TOL, (k, e)


# evaluation of few points per leaf (from the columns) and of many (from the
# Taylor blocks), with derivatives, at one point and at odd remainders; node
# halves beyond 32 (eps 1e-18).  Bars of the derivative routes: 1e-12 for the
# potential, a digit more per derivative.
EVAL_CASES = [  # kind, ns, nt, delta, eps, nd, pgh
    ("uniform", 4000, 1, 2e-2, 1e-6, 1, 3),
    ("uniform", 4001, 7000, 2e-2, 1e-6, 1, 2),
    ("uniform", 2500, 777, 2e-2, 1e-9, 2, 3),
    ("cluster", 9001, 12007, 2e-2, 1e-6, 1, 2),
    ("cluster", 9001, 4003, 2e-2, 1e-12, 1, 1),
    ("uniform", 1200, 901, 5e-2, 1e-18, 1, 2),
]


@pytest.mark.parametrize("case", EVAL_CASES, ids=[f"{c[0]}_{c[4]:g}_{c[2]}_{c[6]}" for c in EVAL_CASES])
def test_sep3d_evaluation(fgt, oracle, case):
    kind, ns, nt, delta, eps, nd, pgh = case
    rng = np.random.default_rng(ns + nt)
    src, trg = _points(kind, ns, rng), _points(kind, nt, rng)
    q = rng.standard_normal((ns, nd))
    ctx = fgt.Context(0, precision="fp64")
    got = fgt.transform_pgh(3, nd, delta, eps, src, q, trg, 1, pgh, ctx=ctx)
    ref = oracle.fgt_pgh(3, nd, delta, eps, src, q, trg, 1, pgh)
    for k, tol in (("pot", 1e-12), ("pottarg", 1e-12), ("gradtarg", 1e-11), ("hesstarg", 1e-10)):
        if got[k] is None:
            continue
        e = oracle.derr(ref[k], got[k])
        print(f"{case}: {k} {e:.2e}")
        assert e <= tol, (k, e)


@pytest.mark.parametrize("eps", [1e-3, 1e-6, 1e-12])
def test_expansions_below_the_cut(fgt, oracle, eps):
    rng = np.random.default_rng(5)
    src = _points("cluster", 8000, rng)
    q = rng.standard_normal((8000, 1))
    ctx = fgt.Context(0, precision="fp64")
    plan = fgt.Plan(ctx, 3, 1, 2e-2, eps, src, None, 1, 0)
    plan.execute_host(src, q)
    inf = plan.info()
    T = fgt.HostTree(3, 2e-2, eps, src, src)
    lev, cut = T["ilevel"], max(inf["npwlevel"], 0)
    below = [b for b in range(T["nboxes"]) if lev[b] > cut]
    pick = sorted(rng.choice(below, size=min(60, len(below)), replace=False).tolist())
    mp, _, has = oracle.expansions(3, 1, 2e-2, eps, src, q, None, 1, 0, pick, inf["nexp"])
    got = [plan.expansion("mp", b) for b in pick]
    plan.close()
    n = 0
    for i, b in enumerate(pick):
        scale = np.abs(mp[i]).max() if has[i] else 0.0
        if scale == 0.0:
            continue
        d = got[i]
        assert d is not None
        assert np.abs(d - mp[i]).max() <= TOL * scale, b
        n += 1
    assert n > 10
