"""Without pinned memory for the staging ring, large results arrive by plain copies: the same row-major traveltime
grids and the same gradient as with it."""
import numpy as np
import pytest

from eikonalsolvers import Context, Grid2DCart, Grid3DCart

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nsrc", [((523, 511), 3), ((101, 103, 107), 2)], ids=["2D", "3D"])
def test_results_without_the_ring(n, nsrc):
    cls = Grid3DCart if len(n) == 3 else Grid2DCart
    grd = cls(hgrid=0.1, cooinit=(0.0,) * len(n), grsize=n)
    rng = np.random.default_rng(7)
    vel = 2.0 + 0.2 * rng.random(n)
    last = 0.1 * (np.array(n) - 1.0)
    cs = rng.uniform(0.3 * last, 0.7 * last, (nsrc, len(n)))
    rec = [rng.uniform(0.05 * last, 0.95 * last, (4, len(n))) for _ in range(nsrc)]
    obs, std = [np.full(4, 1.0)] * nsrc, [np.full(4, 0.1)] * nsrc
    ctx = Context(0)
    try:
        mid = ctx.upload(vel, grd)
        out = []
        for ring in (1.0, 0.0, 1.0):
            ctx.set_param("host_ring", ring)
            picks, tts = ctx.traveltime(mid, grd, cs, rec, returntt=True)
            out.append([*picks, *tts, ctx.gradient(mid, grd, cs, rec, obs, std, "gradvel")[0]])
    finally:
        ctx.close()
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], o))
