"""Sharded plans whose ranks differ in density: the kernels of an order and
the sources per partial block follow from the points of all ranks, so the sum
of the ranks' outputs equals the one-GPU result bit for bit here too.  Each
case has one rank whose own points alone would choose otherwise: a lower half
(in the last coordinate) denser than the upper one, or a ball that holds half
the points (a leaf of more than one partial block)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, h, per):
    """n coordinates, per of them in every box of side h, about zero."""
    return (np.arange(n) - (n - 1) / 2) * h / per


def _evaluation_72(rng):
    # order 30, leaves of 76 sources below and 25 above: k_eval2d_mma or Horner
    h = math.sqrt(1e-4 * math.log(1e9)) / 2
    x = _rows(2 * int(4 / h), h, 8.0)
    y = np.concatenate([_rows(2 * int(2.4 / h), h, 9.5), _rows(2 * int(0.8 / h), h, 3.0)])
    y[2 * int(2.4 / h):] += _rows(2 * int(2.4 / h), h, 9.5)[-1] + 0.5 * h - _rows(2 * int(0.8 / h), h, 3.0)[0]
    p = np.stack(np.meshgrid(x, y), -1).reshape(-1, 2)
    return p + (rng.random(p.shape) - 0.5) * 0.02 * h


def _formation_80(rng):
    # order 18, leaves of about 115 sources below and 22 above: a CTA or a warp per leaf
    out = []
    for half, m in enumerate((300, 130)):
        g = np.stack(np.meshgrid((np.arange(m) + 0.5) / m, (np.arange(m // 2) + 0.5) / (m // 2)), -1).reshape(-1, 2)
        g = g + (rng.random(g.shape) - 0.5) * 0.5 / m
        g[:, 1] = 0.5 * (g[:, 1] + half)
        out.append(g)
    return np.concatenate(out)


def _halves(n0, n1):
    def make(rng):
        a, b = rng.random((n0, 3)), rng.random((n1, 3))
        a[:, 2] *= 0.5
        b[:, 2] = 0.5 + 0.5 * b[:, 2]
        return np.concatenate([a, b])
    return make


def _ball(dim, n):
    def make(rng):
        x = rng.random((n, dim))
        x[:n // 2] = 0.37 + 1e-5 * x[:n // 2]
        return x
    return make


CASES = [
    ("evaluation_72", 2, 1e-4, 1e-9, _evaluation_72, 1, "fp64"),
    ("formation_80", 2, 1e-3, 1e-9, _formation_80, 1, "fp64"),
    ("blocks_or_columns", 3, 1e-2, 1e-6, _halves(147000, 15000), 2, "fp64"),
    ("chunk_2d", 2, 1e-3, 1e-6, _ball(2, 1300000), 1, "fp64"),
    ("chunk_2d", 2, 1e-3, 1e-6, _ball(2, 1300000), 1, "mixed"),
    ("chunk_3d", 3, 1e-2, 1e-6, _ball(3, 600000), 1, "fp64"),
]


@pytest.mark.parametrize("name,dim,delta,eps,points,pgh,precision", CASES, ids=[f"{c[0]}-{c[6]}" for c in CASES])
def test_ranks_of_unequal_density(fgt, name, dim, delta, eps, points, pgh, precision):
    import torch
    from fgt2d_b200.shard import ShardPlan
    rng = np.random.default_rng(31)
    src = np.ascontiguousarray(points(rng))
    n, R = src.shape[0], 2
    dev = torch.device("cuda", 0)
    ctx = fgt.Context(0, precision=precision)
    q = torch.from_numpy(rng.standard_normal((n, 1))).to(dev)
    one = fgt.Plan(ctx, dim, 1, delta, eps, src, None, pgh, 0)
    ref = torch.zeros((n, 1), dtype=torch.float64, device=dev)
    one.execute_device(0, q.data_ptr(), 0, ref.data_ptr(), 0)
    plans = [ShardPlan(ctx, dim, 1, delta, eps, src, None, pgh, 0, R, r) for r in range(R)]
    out = [torch.full((n, 1), np.nan, dtype=torch.float64, device=dev) for _ in plans]
    for p, o in zip(plans, out):
        p.phase(1, q.data_ptr(), o.data_ptr(), 0)
    torch.cuda.synchronize()
    for r, p in enumerate(plans):
        ns, _ = p.counts(1 - r)
        if ns:
            buf = torch.empty(ns * p.slot_doubles(), dtype=torch.float64, device=dev)
            p.pack(1 - r, buf.data_ptr())
            torch.cuda.synchronize()
            plans[1 - r].unpack(r, buf.data_ptr())
            torch.cuda.synchronize()
    for p, o in zip(plans, out):
        p.phase(2, q.data_ptr(), o.data_ptr(), 0)
    torch.cuda.synchronize()
    for p in plans:
        p.close()
    one.close()
    assert torch.equal(out[0] + out[1], ref)
