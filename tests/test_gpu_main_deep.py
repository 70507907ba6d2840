"""A caller's tree (fgt2dmain_gpu_ / fgt3dmain_gpu_) with leaves far below the
cut level: the box at the origin's corner refined at every level, a few points
in every leaf.  8 and 9 levels are the edge between phase rows for every place
and for those that occur; 40 are more than a table of every place could hold.

Against the direct sum: ten times the precision asked for."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_ip = ctypes.POINTER(ctypes.c_int)
_lp = ctypes.POINTER(ctypes.c_longlong)
_dp = ctypes.POINTER(ctypes.c_double)


def _tree(dim, levels):
    """The chain: per level the 2^dim children of the corner box, in the
    reference's arrays, and the leaves in the order of their points."""
    nch, nco = 2 ** dim, 3 ** dim
    nb = 1 + nch * levels
    first = [1] + [2 + nch * (lev - 1) for lev in range(1, levels + 1)]  # 1-based
    laddr = np.array([[first[lev], first[lev] + (nch if lev else 1) - 1] for lev in range(levels + 1)], dtype=np.int32)
    lev, par = np.zeros(nb, np.int32), np.full(nb, -1, np.int32)
    nchild, child = np.zeros(nb, np.int32), np.full((nb, nch), -1, np.int32)
    nnb, nbr = np.ones(nb, np.int32), np.full((nb, nco), -1, np.int32)
    cen = np.full((nb, dim), 0.5)
    nbr[0, 0] = 1
    for k in range(1, levels + 1):
        p = first[k - 1]  # the corner box of the level above
        nchild[p - 1] = nch
        for j in range(nch):
            b = first[k] + j
            child[p - 1, j], par[b - 1], lev[b - 1] = b, p, k
            sign = np.array([1.0 if j >> d & 1 else -1.0 for d in range(dim)])
            cen[b - 1] = cen[p - 1] + sign * 0.5 ** (k + 1)
            nnb[b - 1] = nch
            nbr[b - 1, :nch] = first[k] + np.arange(nch)
    leaves = [first[levels]] + [first[k] + j for k in range(levels, 0, -1) for j in range(1, nch)]
    return first, laddr, lev, par, nchild, child, nnb, nbr, cen, leaves


@pytest.mark.parametrize("levels", [8, 9, 40])
@pytest.mark.parametrize("dim,per", [(2, 7), (3, 3)])
def test_deep_tree(fgt, oracle, dim, levels, per):
    eps = 1e-9
    delta = 1.0 / math.log(1.0 / eps)  # the root box is the cut level's
    first, laddr, lev, par, nchild, child, nnb, nbr, cen, leaves = _tree(dim, levels)
    nb = lev.size
    rng = np.random.default_rng(levels + dim)
    src = np.concatenate([cen[b - 1] + (rng.random((per, dim)) - 0.5) * 0.5 ** int(lev[b - 1]) for b in leaves])
    trg = np.concatenate([cen[b - 1] + (rng.random((per, dim)) - 0.5) * 0.5 ** int(lev[b - 1]) for b in leaves])
    n = src.shape[0]
    q = rng.standard_normal(n)
    se = np.zeros((nb, 2), np.int32)
    for i, b in enumerate(leaves):
        se[b - 1] = per * i + 1, per * (i + 1)
    for k in range(levels - 1, -1, -1):  # a corner box holds the points of its children
        se[first[k] - 1] = 1, se[child[first[k] - 1] - 1, 1].max()
    parts = [laddr.ravel(), lev, par, nchild, child.ravel(), nnb, nbr.ravel()]
    iptr = np.cumsum([1] + [a.size for a in parts]).astype(np.int64)
    itree = np.concatenate(parts).astype(np.int32)
    boxsize = 0.5 ** np.arange(levels + 1)
    nlocal = np.array([oracle.hlterms(dim, b, delta, eps) for b in boxsize], dtype=np.int32)
    pmax, npw = oracle.pwterms(2.0, delta, eps)
    pot, pt = np.zeros(n), np.zeros(n)
    dummy, iaddr = np.zeros(2), np.zeros(2, dtype=np.int32)
    P = lambda a: a.ctypes.data_as(_dp)
    I = lambda a: a.ctypes.data_as(_ip)
    i = lambda v: ctypes.byref(ctypes.c_int(v))
    d = lambda v: ctypes.byref(ctypes.c_double(v))
    common = [i(1), d(delta), d(eps), i(n), P(src), i(1), P(q), i(0), P(dummy), P(dummy), i(n), P(trg), I(iaddr),
              P(dummy), I(itree)]
    tail = [i(nb), i(0), P(boxsize), P(cen), I(laddr), I(se), I(se), I(nlocal), I(nlocal), i(int(nlocal.max())),
            d(pmax), i(npw), i(1), P(pot), P(dummy), P(dummy), i(1), P(pt), P(dummy), P(dummy)]
    L = fgt.lib()
    if dim == 2:
        st = L.fgt2dmain_gpu_(*common, i(itree.size), I(iptr.astype(np.int32)), i(levels), i(0), *tail)
    else:
        st = L.fgt3dmain_gpu_(*common, ctypes.byref(ctypes.c_longlong(itree.size)), iptr.ctypes.data_as(_lp),
                              i(levels), i(0), i(100), *tail)
    assert st == 0
    assert oracle.derr(oracle.direct(dim, 1, delta, src, q, src)[:, 0], pot) <= 10 * eps
    assert oracle.derr(oracle.direct(dim, 1, delta, src, q, trg)[:, 0], pt) <= 10 * eps
