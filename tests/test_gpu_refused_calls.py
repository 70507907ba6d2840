"""Calls that are refused for a value that is not finite, at sizes on either
side of the smallest tree built on the device: the same status, and the
drop-in call's outputs are zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", ["charge", "source", "target", "dipole"])
@pytest.mark.parametrize("n", [1, 500, 5000])
@pytest.mark.parametrize("tree", [None, "host"])
def test_refused_call_zeroes_its_outputs(fgt, bad, n, tree):
    rng = np.random.default_rng(n)
    src, trg, q = rng.random((n, 2)), rng.random((n, 2)), rng.random((n, 1))
    rn, ds = rng.random((n, 2)), rng.random((n, 1))
    {"charge": q, "source": src, "target": trg, "dipole": ds}[bad][n // 2, 0] = np.nan
    ctx = fgt.Context(0) if tree is None else fgt.Context(0, tree=tree)
    out = {k: np.full(s, 7.0) for k, s in (("pot", (n, 1)), ("grad", (n, 2, 1)), ("pottarg", (n, 1)))}
    with pytest.raises(fgt.FGTError) as e:
        fgt.transform_pgh(2, 1, 1e-3, 1e-6, src, q, trg, 2, 1, ctx, 1, 1, rn, ds, out)
    assert e.value.status == 1
    for k, v in out.items():
        assert np.all(v == 0.0), k


def test_no_sources(fgt):
    """Without sources the fields are zero, whatever the targets hold."""
    trg = np.full((10, 2), np.nan)
    ctx = fgt.Context(0)
    _, pt = fgt.transform(2, 1, 1e-3, 1e-6, np.zeros((0, 2)), np.zeros((0, 1)), trg, 0, 1, ctx=ctx)
    assert np.all(pt == 0.0)
