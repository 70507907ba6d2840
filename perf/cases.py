"""What the transform is used for, as cases that can be timed and compared.

Two ways of using the library are covered, each through the public package:

* ``plan``: a program that keeps the points (a time stepper, an iterative
  solver, a density estimate over many weight vectors) builds a ``Plan`` once
  and applies it to new charges that are on the GPU already;
* ``call``: the drop-in call, host arrays in and host arrays out, with the
  tree built inside (``transform_pgh``, the replacement of the Fortran
  ``call fgt2d`` / ``call fgt3d``).

A case is a dict of plain values: ``entry``, ``dim``, ``dist`` ("uniform" in
the unit box; "circle": 2D, 90% on a circle of radius 0.3 with radial jitter
1e-3; "blobs": 3D, 80% in 16 Gaussian blobs of width 0.02), ``ns`` sources and
``nt`` separate targets (0: none), ``nd`` densities, ``delta``, ``eps``, the
output levels ``pgh`` at the sources and ``pght`` at the targets (1
potential, 2 with gradient, 3 with Hessian), and ``dipoles`` beside the
charges.  The precision is the library's default: mixed arithmetic from eps
1e-6 up, FP64 below.
"""
import math

import numpy as np
import torch

import fgt2d_b200 as fgt

DEV = "cuda:0"
F64 = torch.float64
_session = {}


def _case(name, entry, dim, dist, ns, delta, eps, nt=0, nd=1, pgh=1, pght=0, dipoles=False):
    c = dict(entry=entry, dim=dim, dist=dist, ns=ns, nt=nt, nd=nd, delta=delta, eps=eps, pgh=pgh, pght=pght,
             dipoles=dipoles)
    return c if name is None else dict(name=name, **c)


def listed():
    return [
        # the smallest requests of a mixed stream: a few hundred to a few
        # thousand points, no far field, launch and call latency only
        _case("call_2d_1e3", "call", 2, "uniform", 1000, 1e-3, 1e-6),
        _case("plan_2d_2e3", "plan", 2, "uniform", 2000, 1e-3, 1e-6),
        # a medium drop-in call: a 3D particle set handed over from host code
        _case("call_3d_1e5", "call", 3, "uniform", 100_000, 1e-3, 1e-6),
        # the drop-in call at the size of the headline benchmark
        _case("call_2d_circle_1e7", "call", 2, "circle", 10_000_000, 1e-6, 1e-6),
        # the headline benchmark: strongly clustered points, charges resident
        _case("plan_2d_circle_1e7", "plan", 2, "circle", 10_000_000, 1e-6, 1e-6),
        # separate targets at high precision, both sets evaluated
        _case("plan_2d_1e5_e9", "plan", 2, "uniform", 100_000, 1e-4, 1e-9, nt=100_000, pght=1),
        # potential, gradient and Hessian at odd sizes: Newton steps on a kernel density
        _case("plan_2d_hess_e9", "plan", 2, "uniform", 300_007, 1e-4, 1e-9, nt=100_003, pgh=3, pght=3),
        # charges and dipoles, two densities: a layer potential of the heat kernel
        _case("plan_2d_dipole_e9", "plan", 2, "uniform", 200_003, 1e-4, 1e-9, nd=2, dipoles=True),
        # the large 3D workload: clustered sources, potentials at separate targets
        _case("plan_3d_blobs_4e6", "plan", 3, "blobs", 4_000_000, 1e-3, 1e-6, nt=4_000_000, pgh=0, pght=1),
        # forces between clustered particles
        _case("plan_3d_force_3e5", "plan", 3, "blobs", 300_000, 1e-3, 1e-6, pgh=2),
        # 3D at the tighter precisions of the precision sweep
        _case("plan_3d_3e5_e9", "plan", 3, "uniform", 300_000, 1e-3, 1e-9),
        _case("plan_3d_3e5_e12", "plan", 3, "uniform", 300_000, 1e-2, 1e-12),
    ]


def draw(rng):
    def logu(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    dim = rng.choice((2, 3))
    entry = rng.choice(("plan", "plan", "plan", "call"))
    eps = rng.choice((1e-3, 1e-6, 1e-6, 1e-9, 1e-12))
    delta = float("%.3g" % logu(1e-6 if dim == 2 else 1e-4, 1e-1))
    # each derivative costs about a digit: no Hessians at three digits
    pgh = rng.choice((1, 1, 1, 1, 2, 2, 3 if eps < 1e-3 else 1))
    # 3D expansions grow as eps^-3 in their terms: sizes that fit three plans
    # on one card and cost no more than the largest listed case
    if dim == 2:
        most = 3_000_000 if pgh == 1 else 1_000_000
    elif eps >= 1e-6:
        most = 1_000_000 if pgh == 1 else 150_000
    else:
        most = 100_000 if pgh == 1 else 30_000
    ns = int(logu(1000, most))
    sets = rng.choice(("sources", "sources", "both", "targets"))
    nt = 0 if sets == "sources" else int(logu(1000, min(most, 4 * ns)))
    dist = rng.choice(("uniform", "circle" if dim == 2 else "blobs"))
    nd = rng.choice((1, 1, 1, 2, 3)) if ns + nt <= 100_000 else 1
    dipoles = rng.random() < 0.15 and ns + nt <= 300_000
    return _case(None, entry, dim, dist, ns, delta, eps, nt=nt, nd=nd, pgh=0 if sets == "targets" else pgh,
                 pght=0 if sets == "sources" else pgh, dipoles=dipoles)


def _points(c, n, g):
    x = torch.rand(n, c["dim"], dtype=F64, device=DEV, generator=g)
    if c["dist"] == "circle":
        m = n - n // 10
        th = torch.rand(m, dtype=F64, device=DEV, generator=g) * (2 * math.pi)
        r = 0.3 + 1e-3 * torch.randn(m, dtype=F64, device=DEV, generator=g)
        x[:m, 0] = 0.5 + r * torch.cos(th)
        x[:m, 1] = 0.5 + r * torch.sin(th)
    elif c["dist"] == "blobs":
        m = n - n // 5
        x[:m] = _points.centres[torch.randint(0, 16, (m,), device=DEV, generator=g)]
        x[:m] += 0.02 * torch.randn(m, 3, dtype=F64, device=DEV, generator=g)
    return x[torch.randperm(n, device=DEV, generator=g)].contiguous()


def _inputs(c, seed):
    """Sources, targets, charges, dipole directions and strengths on the GPU."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    _points.centres = torch.rand(16, 3, dtype=F64, device=DEV, generator=g) * 0.8 + 0.1
    src = _points(c, c["ns"], g)
    trg = _points(c, c["nt"], g) if c["nt"] else None
    q = torch.randn(c["ns"], c["nd"], dtype=F64, device=DEV, generator=g)
    rn = ds = None
    if c["dipoles"]:
        rn = torch.randn(c["ns"], c["dim"], dtype=F64, device=DEV, generator=g)
        rn /= rn.norm(dim=1, keepdim=True)
        ds = torch.randn(c["ns"], c["nd"], dtype=F64, device=DEV, generator=g)
    return src, trg, q, rn, ds


def _names(c):
    """(output, points, components) of the outputs that the case asks for."""
    comps = (1, c["dim"], fgt.nhess(c["dim"]))
    got = []
    for n, pgh, names in ((c["ns"], c["pgh"], ("pot", "grad", "hess")),
                          (c["nt"], c["pght"], ("pottarg", "gradtarg", "hesstarg"))):
        got += [(names[i], n, comps[i]) for i in range(pgh)]
    return got


def _shape(c, n, k):
    return (n, c["nd"]) if k == 1 else (n, k, c["nd"])


def prepare(case, seed):
    c = case
    if not _session:
        # one context and one stream for the whole program
        _session["ctx"] = fgt.Context(0)
        _session["stream"] = torch.cuda.Stream(DEV)
    src, trg, q, rn, ds = _inputs(c, seed)
    s = dict(case=c)
    if c["entry"] == "call":
        def host(t):
            return None if t is None else t.cpu().pin_memory().numpy()

        s.update(src=host(src), trg=host(trg), q=host(q), rn=host(rn), ds=host(ds))
        s["out"] = {k: torch.zeros(_shape(c, n, m), dtype=F64).pin_memory().numpy() for k, n, m in _names(c)}
    else:
        s["plan"] = fgt.Plan(_session["ctx"], c["dim"], c["nd"], c["delta"], c["eps"], src.cpu().numpy(),
                             None if trg is None else trg.cpu().numpy(), c["pgh"], c["pght"], 1, int(c["dipoles"]))
        s.update(q=q, rn=rn, ds=ds)
        s["out"] = {k: torch.zeros(_shape(c, n, m), dtype=F64, device=DEV) for k, n, m in _names(c)}
    torch.cuda.synchronize()
    return s


def run(state):
    c, out = state["case"], state["out"]
    if c["entry"] == "call":
        fgt.transform_pgh(c["dim"], c["nd"], c["delta"], c["eps"], state["src"], state["q"], state["trg"], c["pgh"],
                          c["pght"], _session["ctx"], 1, int(c["dipoles"]), state["rn"], state["ds"], out)
        return out
    stream = _session["stream"].cuda_stream
    plan = state["plan"]

    def ptr(t):
        return 0 if t is None else t.data_ptr()

    o = [ptr(out.get(k)) for k in ("pot", "grad", "hess", "pottarg", "gradtarg", "hesstarg")]
    if c["dipoles"]:
        st = fgt.lib().fgt_plan_execute_device_full(plan._h, ptr(state["q"]), ptr(state["rn"]), ptr(state["ds"]),
                                                    *[p or None for p in o], stream)
        if st:
            raise fgt.FGTError(st, "fgt_plan_execute_device_full")
    elif max(c["pgh"], c["pght"]) >= 2:
        plan.execute_device_pgh(ptr(state["q"]), *o, stream=stream)
    else:
        plan.execute_device(0, ptr(state["q"]), 0, o[0], o[3], stream=stream)
    return out


def work(case):
    c = case
    # an expansion term costs one multiply-add per source and one per point and
    # component; about 2 digits + 1 terms per dimension.  Where fewer sources
    # than terms lie within reach of a point, their direct sum is what remains.
    terms = (2 * round(-math.log10(c["eps"])) + 1) ** c["dim"]
    reach = math.sqrt(c["delta"] * math.log(1 / c["eps"]))
    ball = math.pi * reach ** 2 if c["dim"] == 2 else 4 / 3 * math.pi * reach ** 3
    each = min(terms, max(1.0, c["ns"] * min(1.0, ball)))
    values = sum(n * k for _, n, k in _names(c))
    flops = 2.0 * c["nd"] * each * (c["ns"] * (2 if c["dipoles"] else 1) + values)
    read = c["ns"] * (c["dim"] + c["nd"]) + c["nt"] * c["dim"] + (c["ns"] * (c["dim"] + c["nd"]) if c["dipoles"] else 0)
    return {"bytes": 8.0 * (read + values * c["nd"]), "flops": flops}


def exact(case, seed):
    """The direct sums, up to 3e11 pairs."""
    c = case
    pairs = c["ns"] * ((c["ns"] if c["pgh"] else 0) + (c["nt"] if c["pght"] else 0))
    if pairs > 3e11 or (c["dipoles"] and max(c["pgh"], c["pght"]) > 1):
        return None
    dim, nd, delta = c["dim"], c["nd"], c["delta"]
    src, trg, q, rn, ds = _inputs(c, seed)
    centre = src.mean(dim=0)
    src = src - centre
    hpairs = [(0, 0), (0, 1), (1, 1)] if dim == 2 else [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    # K @ W gives the sums of q, q s_a and q s_a s_b that the derivatives need;
    # a dipole adds the vectors v = dipstr n and v . s
    level = max(c["pgh"], c["pght"])
    cols = [q]
    if level >= 2:
        cols += [q * src[:, a:a + 1] for a in range(dim)]
    if level >= 3:
        cols += [q * src[:, a:a + 1] * src[:, b:b + 1] for a, b in hpairs]
    if c["dipoles"]:
        v = [ds * rn[:, a:a + 1] for a in range(dim)]
        cols += v + [sum(v[a] * src[:, a:a + 1] for a in range(dim))]
    weights = torch.cat(cols, dim=1)
    got = {}
    for pts, pgh, names in ((src, c["pgh"], ("pot", "grad", "hess")),
                            (None if trg is None else trg - centre, c["pght"], ("pottarg", "gradtarg", "hesstarg"))):
        if not pgh:
            continue
        parts = [[] for _ in range(pgh)]
        step = max(1, int(2.5e8) // c["ns"])
        for t0 in range(0, pts.shape[0], step):
            x = pts[t0:t0 + step]
            kern = None
            for a in range(dim):
                d = x[:, a:a + 1] - src[None, :, a]
                d.mul_(d)
                kern = d if kern is None else kern.add_(d)
            m = (kern.mul_(-1.0 / delta).exp_() @ weights).reshape(x.shape[0], -1, nd)
            pot = m[:, 0]
            if c["dipoles"]:
                # 2 / delta sum K v . (x - s)
                pot = pot + 2 / delta * (sum(x[:, a:a + 1] * m[:, 1 + a] for a in range(dim)) - m[:, 1 + dim])
            parts[0].append(pot)
            first = [x[:, a:a + 1] * m[:, 0] - m[:, 1 + a] for a in range(dim)] if pgh >= 2 else []
            if pgh >= 2:
                parts[1].append(torch.stack([-2 / delta * f for f in first], dim=1))
            if pgh >= 3:
                h = []
                for i, (a, b) in enumerate(hpairs):
                    xa, xb = x[:, a:a + 1], x[:, b:b + 1]
                    second = xa * xb * m[:, 0] - xa * m[:, 1 + b] - xb * m[:, 1 + a] + m[:, 1 + dim + i]
                    h.append(4 / delta ** 2 * second - (2 / delta * m[:, 0] if a == b else 0.0))
                parts[2].append(torch.stack(h, dim=1))
        for k in range(pgh):
            got[names[k]] = torch.cat(parts[k])
    return got
