"""Timed workloads of the forward and adjoint paths, through the package's public entry points.

Every case is one call as a user's program makes it: host arrays in, host arrays out, on a
context that already holds the velocity model (or, for the one-shot functions, uploads it
in the call), with the launch parameters the shipped autotuner table has for its class.
"""
import heapq
import math
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.getcwd(), "eikonalsolvers.jl_b200"))

from eikonalsolvers import (Context, ExtraParams, Grid2DCart, Grid2DSphere, Grid3DCart,  # noqa: E402
                            Grid3DSphere, eiktraveltime)
from eikonalsolvers import configs  # noqa: E402
from eikonalsolvers.tune import default_tuner  # noqa: E402


def _case(name, call, grid, n, nsrc, nrec, model, which="", returntt=False, refine=True, smooth=0):
    c = dict(call=call, grid=grid, n1=n[0], n2=n[1], n3=n[2] if len(n) == 3 else 0, nsrc=nsrc, nrec=nrec,
             model=model, which=which, returntt=returntt, refine=refine, smooth=smooth)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # smallest call: one source on a small section, latency of a single forward solve
        _case("tt2d_one", "traveltime", "cart", (128, 80), 1, 10, "gradient", returntt=True),
        # the reference's own kind of call: one-shot function, whole traveltime grids wanted
        _case("tt2d_oneshot", "oneshot", "cart", (300, 220), 4, 10, "gradient", returntt=True),
        # a sampler: the captured pipeline replayed with a new velocity at every evaluation
        _case("plan2d_sampler", "plan", "cart", (300, 220), 4, 10, "random", which="gradvel"),
        # 2D inversion step: random-field model, many sources, receivers along the surface
        _case("grad2d_survey", "gradient", "cart", (1024, 640), 64, 200, "random", which="gradvel"),
        # 2D polar section of odd size, summed gradient smoothed
        _case("grad2d_sphere", "gradient", "sphere", (181, 241), 9, 37, "gradient", which="gradvel", smooth=5),
        # serving: traveltime requests on three models of different size merged into one call
        _case("multi2d_serving", "multi", "cart", (517, 323), 26, 10, "random"),
        # small 3D box without the refined start-up, source locations wanted
        _case("srcloc3d_box", "gradient", "cart", (44, 44, 44), 16, 40, "layered", which="gradsrcloc", refine=False),
        # 3D inversion step on a small grid
        _case("grad3d_small", "gradient", "cart", (64, 64, 64), 32, 100, "layered", which="gradvelandsrcloc"),
        # ragged 3D grid, a few sources, picks only
        _case("tt3d_ragged", "traveltime", "cart", (151, 97, 203), 5, 61, "random"),
        # one event alone on a 3D grid: nothing to batch
        _case("grad3d_single", "gradient", "cart", (128, 128, 128), 1, 100, "layered", which="gradvelandsrcloc"),
        # regional inversion step on a spherical box
        _case("grad3d_sphere", "gradient", "sphere", (100, 90, 90), 12, 500, "random", which="gradvel"),
        # large 3D inversion step: velocity and source-location gradients
        _case("grad3d_large", "gradient", "cart", (256, 256, 256), 4, 400, "layered", which="gradvelandsrcloc"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["traveltime", "traveltime", "gradient", "gradient", "gradient", "oneshot", "plan", "multi"])
    grid = "sphere" if call in ("traveltime", "gradient") and rng.random() < 0.3 else "cart"
    three = call != "multi" and rng.random() < 0.55
    if three:
        most = {"plan": 64, "oneshot": 128}.get(call, 224)
        side = _logint(rng, 24, most)
        n = tuple(max(12, int(side * rng.uniform(0.6, 1.2))) for _ in range(3))
        cap = 40_000_000 if grid == "cart" else 9_000_000
    else:
        side = _logint(rng, 64, 512 if call in ("plan", "oneshot") else 1024)
        n = (side, max(24, int(side * rng.uniform(0.5, 1.0))))
        cap = 32_000_000
    npts = math.prod(n)
    nsrc = max(1, min(_logint(rng, 1, 64), cap // npts))
    if call == "plan":
        nsrc = min(nsrc, 16)
    returntt = call in ("traveltime", "oneshot") and rng.random() < 0.4
    if returntt:
        nsrc = min(nsrc, 30, max(1, 8_000_000 // npts))
    which = ""
    if call in ("gradient", "plan"):
        which = "gradvel" if grid == "sphere" else rng.choice(["gradvel", "gradsrcloc", "gradvelandsrcloc"])
    nrec = _logint(rng, 5, 400)
    model = rng.choice(["gradient", "random", "layered"] if three and grid == "cart" else ["gradient", "random"])
    smooth = rng.choice([0, 0, 5]) if "vel" in which else 0
    return _case("", call, grid, n, nsrc, nrec, model, which, returntt, rng.random() < 0.8, smooth)


def _dims(case):
    return (case["n1"], case["n2"], case["n3"]) if case["n3"] else (case["n1"], case["n2"])


def _grid(case, n):
    if case["grid"] == "cart":
        cls = Grid3DCart if len(n) == 3 else Grid2DCart
        return cls(hgrid=0.1 if len(n) == 3 else 0.25, cooinit=(0.0,) * len(n), grsize=n)
    dr, da = 600.0 / (n[0] - 1), [20.0 / (m - 1) for m in n[1:]]
    if len(n) == 3:
        return Grid3DSphere(Δr=dr, Δθ=da[0], Δφ=da[1], cooinit=(5771.0, 80.0, 80.0), grsize=n)
    return Grid2DSphere(Δr=dr, Δθ=da[0], cooinit=(5771.0, 80.0), grsize=n)


def _velocity(case, n, seed):
    depth = np.linspace(0.0, 1.0, n[0] if case["grid"] == "sphere" else n[-1])
    if case["grid"] == "sphere":
        depth = (1.0 - depth).reshape((-1,) + (1,) * (len(n) - 1))
    lo, hi = (5.8, 8.0) if case["grid"] == "sphere" else (2.5, 2.5 + 0.01 * n[-1])
    vel = np.broadcast_to(lo + (hi - lo) * depth, n)
    if case["model"] == "layered":
        vel = configs.layered_3d(n, seed=seed)
    elif case["model"] == "random":
        f = configs.gaussian_random_field(n, 20.0 if len(n) == 2 else 6.0, seed)
        vel = vel * (1.0 + 0.03 * f) if case["grid"] == "sphere" else 3.5 + 1.5 * np.tanh(f)
    return np.ascontiguousarray(vel, dtype=np.float64)


def _survey(case, grd, n, nsrc, rng):
    """Sources inside the model (off the nodes), receivers spread over its surface."""
    nd = len(n)
    first = [ax[0] for ax in _axes(grd, nd)]
    last = [ax[-1] for ax in _axes(grd, nd)]
    lo = [a + 0.08 * (b - a) for a, b in zip(first, last)]
    hi = [a + 0.92 * (b - a) for a, b in zip(first, last)]
    surf = 0 if case["grid"] == "sphere" else nd - 1
    cs = np.column_stack([rng.uniform(lo[d], hi[d], nsrc) for d in range(nd)])
    rec = [np.column_stack([np.full(case["nrec"], last[0] if case["grid"] == "sphere" else first[d]) if d == surf
                            else rng.uniform(first[d], last[d], case["nrec"]) for d in range(nd)])
           for _ in range(nsrc)]
    return cs, rec


def _axes(grd, nd):
    names = ("r", "θ", "φ") if isinstance(grd, (Grid2DSphere, Grid3DSphere)) else ("x", "y", "z")
    return [getattr(grd, a) for a in names[:nd]]


def _distance(grd, rec, src):
    if isinstance(grd, (Grid2DCart, Grid3DCart)):
        return np.linalg.norm(rec - src, axis=1)
    def xyz(p):
        p = np.atleast_2d(p)
        th = np.deg2rad(p[:, 1])
        if p.shape[1] == 2:
            return np.column_stack([p[:, 0] * np.cos(th), p[:, 0] * np.sin(th)])
        ph = np.deg2rad(p[:, 2])
        return np.column_stack([p[:, 0] * np.sin(th) * np.cos(ph), p[:, 0] * np.sin(th) * np.sin(ph),
                                p[:, 0] * np.cos(th)])
    return np.linalg.norm(xyz(rec) - xyz(src), axis=1)


def _inputs(case, seed):
    n = _dims(case)
    rng = np.random.default_rng([seed, 17])
    grd, vel = _grid(case, n), _velocity(case, n, seed)
    cs, rec = _survey(case, grd, n, case["nsrc"], rng)
    ep = ExtraParams(refinearoundsrc=case["refine"], smoothgradkern=case["smooth"])
    return n, rng, grd, vel, cs, rec, ep


def prepare(case, seed):
    n, rng, grd, vel, cs, rec, ep = _inputs(case, seed)
    ctx = Context(0)
    default_tuner().apply_known(ctx, grd, case["nsrc"], ep)
    st = dict(call=case["call"], ctx=ctx, grd=grd, vel=vel, cs=cs, rec=rec, ep=ep, which=case["which"],
              returntt=case["returntt"])
    if case["call"] in ("gradient", "plan"):
        # straight-ray times at the mean velocity plus noise stand for the observed picks
        vm = float(vel.mean())
        st["obs"] = [_distance(grd, r, c) / vm + rng.normal(0.0, 0.01, len(r)) for r, c in zip(rec, cs)]
        st["std"] = [np.full(len(r), 0.01) for r in rec]
    if case["call"] == "multi":
        # three resident models, the sources split over them
        left = case["nsrc"]
        st["requests"] = []
        for k, part in enumerate((0.5, 0.3, 0.2)):
            nk = tuple(max(24, int(m * (1.0, 0.7, 0.4)[k])) for m in n)
            ns = left if k == 2 else min(left, max(1, int(case["nsrc"] * part)))
            left -= ns
            if ns == 0:
                continue
            gk = _grid(case, nk)
            ck, rk = _survey(case, gk, nk, ns, rng)
            st["requests"].append((ctx.upload(_velocity(case, nk, seed + k), gk), gk, ck, rk))
    elif case["call"] != "oneshot":
        st["model"] = ctx.upload(vel, grd)
    if case["call"] == "plan":
        st["plan"] = ctx.plan_gradient(st["model"], grd, cs, rec, case["which"], extraparams=ep)
        st["vel"] = vel * (1.0 + 0.01 * rng.uniform(-1.0, 1.0, n))
    return st


def run(state):
    s, call = state, state["call"]
    if call == "traveltime":
        return s["ctx"].traveltime(s["model"], s["grd"], s["cs"], s["rec"], s["returntt"], s["ep"])
    if call == "oneshot":
        return eiktraveltime(s["vel"], s["grd"], s["cs"], s["rec"], s["returntt"], s["ep"], ctx=s["ctx"])
    if call == "gradient":
        return s["ctx"].gradient(s["model"], s["grd"], s["cs"], s["rec"], s["obs"], s["std"], s["which"], s["ep"])
    if call == "plan":
        return s["plan"].run(s["obs"], s["std"], vel=s["vel"])
    return s["ctx"].traveltime_multi(s["requests"], extraparams=s["ep"])


def work(case):
    """Forward: the velocity read and the traveltime written at every node for every source, one
    2nd-order update (~60 flops) each. Gradient: the traveltimes read back and the adjoint
    field written on top, one row of the transposed system (~50 flops) each."""
    npts = math.prod(_dims(case))
    nodes = npts * case["nsrc"]
    if case["call"] == "multi":
        nodes = nodes * (0.5 + 0.3 * 0.49 + 0.2 * 0.16)
    grad = case["call"] in ("gradient", "plan")
    return {"bytes": (32.0 if grad else 16.0) * nodes, "flops": (110.0 if grad else 60.0) * nodes}


# ------------------------------------------------------------- plain restatement --
# The 2nd-order fast-marching solve of a 2D Cartesian model in plain Python floats (64 bits),
# with the refined grid around the source. Small cases only: a node costs tens of
# microseconds here. Gradients have no entry: their plain form is the whole discrete adjoint.

def _local(tt, acc, n, i, j, h, slow):
    alpha, beta, gamma = 0.0, 0.0, -(slow * slow)
    firsts = []
    for ax in (0, 1):
        c1 = c2 = None
        for sh in (1, -1):
            p = (i + sh, j) if ax == 0 else (i, j + sh)
            if not (0 <= p[0] < n[0] and 0 <= p[1] < n[1]) or not acc[p]:
                continue
            if c1 is not None and tt[p] >= c1:
                continue
            c1 = tt[p]
            q = (i + 2 * sh, j) if ax == 0 else (i, j + 2 * sh)
            if 1 <= p[0] <= n[0] - 2 and 1 <= p[1] <= n[1] - 2 and acc[q]:
                c2 = tt[q] if tt[q] <= c1 else None
        if c1 is None:
            continue
        firsts.append(c1)
        if c2 is not None:
            x, a = (1.0 / 3.0) * (4.0 * c1 - c2), 9.0 / (4.0 * (h * h))
        else:
            x, a = c1, 1.0 / (h * h)
        alpha += a
        beta += (-2.0 * a) * x
        gamma += a * (x * x)
    sq = beta * beta - (4.0 * alpha) * gamma
    if sq < 0.0:  # 1st order on every axis, then along one axis only
        a = 1.0 / (h * h)
        alpha, beta, gamma = 0.0, 0.0, -(slow * slow)
        for x in firsts:
            alpha += a
            beta += (-2.0 * a) * x
            gamma += a * (x * x)
        sq = beta * beta - (4.0 * alpha) * gamma
        if sq < 0.0:
            return h * slow + min(firsts)
    return (-beta + math.sqrt(sq)) / (2.0 * alpha)


def _march(tt, acc, n, h, slow, seeds, on_accept):
    """Accepts nodes in order of traveltime from the seeds until on_accept says stop."""
    cur, heap = {}, []

    def near(p):
        for d in ((1, 0), (0, 1), (-1, 0), (0, -1)):
            q = (p[0] + d[0], p[1] + d[1])
            if 0 <= q[0] < n[0] and 0 <= q[1] < n[1] and not acc[q]:
                yield q

    def put(q):
        cur[q] = _local(tt, acc, n, q[0], q[1], h, slow[q])
        heapq.heappush(heap, (cur[q], q))
    for p in seeds:
        for q in near(p):
            if q not in cur:
                put(q)
    while heap:
        v, popped = heap[0][0], []
        while heap and (heap[0][0] == v or cur.get(heap[0][1]) != heap[0][0]):
            t, p = heapq.heappop(heap)
            if acc[p] or cur.get(p) != t:
                continue
            acc[p], tt[p] = True, t
            if on_accept(p):
                return
            popped.append(p)
        for p in popped:
            for q in near(p):
                put(q)


def _box(x, y, h, n):
    i, j = min(int(x // h), n[0] - 2), min(int(y // h), n[1] - 2)
    return [(i, j), (i + 1, j), (i, j + 1), (i + 1, j + 1)]


def _plain2d(vel, h, src, refine, ds=5, rad=3):
    n = vel.shape
    tt, acc = np.full(n, np.inf), np.zeros(n, dtype=bool)
    slow = 1.0 / vel
    box = _box(src[0], src[1], h, n)
    seeds = []
    if refine:
        a = [max(0, box[0][d] - rad) for d in (0, 1)]
        b = [min(n[d] - 1, box[3][d] + rad) for d in (0, 1)]
        m = tuple((b[d] - a[d]) * ds + 1 for d in (0, 1))
        hf = h / ds
        idx = [np.array([a[d] + k // ds + (1 if (k % ds) + 1 >= ds / 2.0 + 1.0 else 0) for k in range(m[d])])
               for d in (0, 1)]
        vf = vel[np.ix_(idx[0], idx[1])]
        tf, af = np.full(m, np.inf), np.zeros(m, dtype=bool)
        o = [a[d] * h for d in (0, 1)]
        fbox = _box(src[0] - o[0], src[1] - o[1], hf, m)
        for p in fbox:
            tf[p], af[p] = math.hypot(o[0] + p[0] * hf - src[0], o[1] + p[1] * hf - src[1]) / vf[p], True

        def accepted(p):
            if p[0] % ds == 0 and p[1] % ds == 0:
                seeds.append(((a[0] + p[0] // ds, a[1] + p[1] // ds), tf[p]))
            edge = any((p[d] == 0 and box[0][d] - rad >= 0) or (p[d] == m[d] - 1 and box[3][d] + rad <= n[d] - 1)
                       for d in (0, 1))
            return edge and len(seeds) > 0
        for p in fbox:
            if p[0] % ds == 0 and p[1] % ds == 0:
                seeds.append(((a[0] + p[0] // ds, a[1] + p[1] // ds), tf[p]))
        _march(tf, af, m, hf, 1.0 / vf, fbox, accepted)
    else:
        seeds = [(p, math.hypot(p[0] * h - src[0], p[1] * h - src[1]) / vel[p]) for p in box]
    for p, t in seeds:
        tt[p], acc[p] = t, True
    _march(tt, acc, n, h, slow, [p for p, _ in seeds], lambda p: False)
    return tt


def exact(case, seed):
    n = _dims(case)
    if case["call"] not in ("traveltime", "oneshot") or case["grid"] != "cart" or len(n) != 2 \
            or n[0] * n[1] * case["nsrc"] > 24_000:
        return None
    _, _, grd, vel, cs, rec, ep = _inputs(case, seed)
    h = grd.hgrid
    grids = [_plain2d(vel, h, c, ep.refinearoundsrc) for c in cs]
    picks = []
    for tt, r in zip(grids, rec):
        x, y = r[:, 0] / h, r[:, 1] / h
        i, j = np.minimum(x.astype(int), n[0] - 2), np.minimum(y.astype(int), n[1] - 2)
        u, w = x - i, y - j
        picks.append(tt[i, j] * (1 - u) * (1 - w) + tt[i + 1, j] * u * (1 - w) + tt[i, j + 1] * (1 - u) * w
                     + tt[i + 1, j + 1] * u * w)
    return (picks, grids) if case["returntt"] else picks
