"""The server's memory estimate against the library's own: eik_gradient_bytes per source, and budgets that
just hold the estimate."""
import numpy as np
import pytest

from eikonalsolvers import Context, ExtraParams, Grid2DCart, Grid3DCart
from eikonalsolvers.serve import request_bytes

# on whole bricks, one node over, thin, larger and smaller than a refined window
SHAPES = [(16, 16), (17, 33), (9, 300), (200, 150), (8, 8, 8), (9, 9, 9), (5, 5, 200), (64, 64, 64)]


def _grid(n):
    return (Grid3DCart if len(n) == 3 else Grid2DCart)(hgrid=0.5, cooinit=(0.0,) * len(n), grsize=n)


def test_a_batch_counts_its_grids_largest_sizes():
    from eikonalsolvers.serve import Request, batch_bytes
    small, thin = _grid((40, 40)), _grid((3, 500))  # more nodes; more bricks
    models = {"a": (None, small), "b": (None, thin)}
    req = [Request(model=m, kind="traveltime", coordsrc=np.zeros((2, 2)), coordrec=[]) for m in "ab"]
    assert batch_bytes(req, models) >= max(request_bytes(g, 4, "traveltime") for g in (small, thin))
    assert batch_bytes(req[:1], models) == request_bytes(small, 2, "traveltime")


@pytest.mark.gpu
@pytest.mark.parametrize("refine", [True, False], ids=["refined", "plain"])
@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
def test_estimate_is_the_librarys(n, refine):
    grd, ep = _grid(n), ExtraParams(refinearoundsrc=refine)
    nodes = int(np.prod(n))
    ctx = Context(0)
    try:
        mid = ctx.upload(np.full(n, 2.0), grd)
        per = (ctx.gradient_bytes(mid, 3, 4, "gradvelandsrcloc", ep)
               - ctx.gradient_bytes(mid, 2, 4, "gradvelandsrcloc", ep))
        # the estimate has an output field more per source and rounds the records up to 1 KB
        assert 0 <= request_bytes(grd, 1, "gradient", ep) - per <= 8 * nodes + 1024
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(17, 33), (200, 150), (9, 9, 9), (40, 41, 43)], ids=lambda n: "x".join(map(str, n)))
def test_calls_fit_the_estimate(n):
    grd, nsrc = _grid(n), 5
    rng = np.random.default_rng(3)
    ext = 0.5 * (np.array(n) - 1.0)
    cs = rng.uniform(0.2 * ext, 0.8 * ext, (nsrc, len(n)))
    rec = [rng.uniform(0.1 * ext, 0.9 * ext, (4, len(n))) for _ in range(nsrc)]
    vel = 2.0 + rng.random(n)
    obs, std = [np.ones(4)] * nsrc, [np.full(4, 0.1)] * nsrc
    for kind in ("traveltime", "gradient"):
        # the model's two fields and 64 KB for inputs, counters and picks
        ctx = Context(0, hbm_budget=16 * vel.size + request_bytes(grd, nsrc, kind) + (64 << 10))
        try:
            mid = ctx.upload(vel, grd)
            if kind == "traveltime":
                ctx.traveltime(mid, grd, cs, rec)
            else:
                ctx.gradient(mid, grd, cs, rec, obs, std, "gradvelandsrcloc")
                assert ctx.last_stats.chunks == 0  # in one pipeline
        finally:
            ctx.close()
