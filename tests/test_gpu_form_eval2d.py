"""2D calls on either side of 3000 points, whose trees are built on the host
and on the device, against the oracle.

FP64, other orders of summation than the oracle's: relative l2 <= 1e-12 for
the potential, a digit more per derivative, as for every FP64 route.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOLS = (("pot", 1e-12), ("pottarg", 1e-12), ("gradtarg", 1e-11), ("hesstarg", 1e-10))

CASES = [  # kind, ns, nt, delta, eps, nd, dipoles, pgh
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
