"""The counted flops of formation and evaluation against counts from the tree:
blocks and sums per point, transforms once per leaf, per column (2D: row) of
leaves and per slab, not per leaf."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _leaves(fgt, oracle, dim, delta, eps, src):
    """(order, points, root, level, places) of every leaf from the cut level on, and that level."""
    T = fgt.HostTree(dim, delta, eps, src, src[:0])
    lev, cut = T["ilevel"], max(T["npwlevel"], 0)
    cen, par = T["centers"].reshape(-1, dim), T["iparent"] - 1
    se = T["isrcse"].reshape(-1, 2)
    out = []
    for b in np.flatnonzero((T["nchild"] == 0) & (lev >= cut)):
        n = int(se[b, 1] - se[b, 0] + 1)
        if n <= 0:
            continue
        a = b
        while lev[a] > cut:
            a = par[a]
        place = tuple(np.round((cen[b] - cen[a]) / T["boxsize"][lev[b]] * 2).astype(int).tolist())
        out.append((oracle.hlterms(dim, T["boxsize"][lev[b]], delta, eps), n, int(a), int(lev[b]), place))
    return out, cut


@pytest.mark.parametrize("dim,n,delta,eps,nd", [(2, 60000, 1e-4, 1e-6, 1), (2, 40000, 1e-3, 1e-9, 2),
                                                (3, 40000, 2e-2, 1e-6, 1), (3, 60001, 1e-2, 1e-3, 2)])
def test_route_flops(fgt, oracle, dim, n, delta, eps, nd):
    rng = np.random.default_rng(n)
    src = rng.random((n, dim))
    ctx = fgt.Context(0, precision="fp64")
    plan = fgt.Plan(ctx, dim, nd, delta, eps, src, None, 1, 0)
    inf = plan.info()
    plan.close()
    L, cut = _leaves(fgt, oracle, dim, delta, eps, src)
    # a leaf at the cut level is evaluated from its own expansion if its sources are not summed directly
    at_cut = [x for x in L if x[3] == cut]
    L = [x for x in L if x[3] > cut]
    assert len(L) > 100
    w, n2 = inf["npw"], inf["npw"] // 2
    form = ev = 0.0
    rows, slabs = set(), set()
    for p, m, root, lev, place in L:
        P = p + 1
        form += 2 * m * P ** dim
        if dim == 2:
            form += 2 * P * P * n2 + 8 * P * n2
            ev += 2 * P * P * n2 + 8 * P * n2 + 2 * m * P * P
            rows.add((P, root, lev, place[1]))
        else:
            form += 2 * P ** 3 * n2 + 8 * P * P * n2
            rows.add((P, root, lev, place[0], place[1]))
            slabs.add((P, root, lev, place[0]))
    for r in rows:
        P = r[0]
        if dim == 2:
            form += 4 * P * n2 ** 2 + 8 * n2 ** 2
            ev += 4 * P * n2 ** 2 + 16 * n2 ** 2
        else:
            form += 4 * P * P * n2 ** 2 + 8 * P * n2 ** 2
    for s in slabs:
        form += (4 * s[0] + 8) * n2 * n2 * w
    assert inf["form_route_flops"] == pytest.approx(nd * form, rel=1e-12)
    if dim == 2:
        most = ev + sum((2 * P * P * n2 + 8 * P * n2 + 4 * P * n2 ** 2 + 16 * n2 ** 2 + 2 * m * P * P)
                        for P, m in ((x[0] + 1, x[1]) for x in at_cut))
        assert nd * ev * (1 - 1e-12) <= inf["eval_route_flops"] <= nd * most * (1 + 1e-12)
    else:
        assert 0 < inf["eval_route_flops"] < inf["eval_flops"] * nd
