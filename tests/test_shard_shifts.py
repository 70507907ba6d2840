"""The shard statistics count the merges and splits of the subtrees of a rank's
cut-level boxes, and the ranks' counts add up to the one-rank plan's (no GPU)."""
import numpy as np
import pytest


@pytest.mark.parametrize("dim,delta,eps,n,seed", [(2, 1e-3, 1e-6, 60000, 11), (3, 1e-2, 1e-6, 20000, 13)])
@pytest.mark.parametrize("flags", [(1, 1), (1, 0), (0, 1)])
def test_shift_counts(fgt, dim, delta, eps, n, seed, flags):
    from fgt2d_b200.shard import HostShard
    rng = np.random.default_rng(seed)
    src, trg = rng.random((n, dim)), rng.random((n // 7, dim))
    src[: n // 2, 0] *= 0.25
    T = fgt.HostTree(dim, delta, eps, src, trg)
    below = T["ilevel"] > max(T["npwlevel"], 0)
    count = lambda f: (lambda r: r[:, 1] - r[:, 0] + 1)(T[f].reshape(-1, 2))
    ns, nt = count("isrcse"), count("itargse")
    want = int((below & (ns > 0)).sum() + (below & (flags[0] * ns + flags[1] * nt > 0)).sum())
    stats = lambda R, r: HostShard(dim, 1, delta, eps, src, trg, *flags, R, r).stats()["shift_tasks"]
    assert stats(1, 0) == want > 0
    assert sum(stats(3, r) for r in range(3)) == want
