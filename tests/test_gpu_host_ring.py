"""Large results through the pinned staging ring: many small grids, several to a slot and cut at its end, are the
column-major ones; and without pinned memory for the ring plain copies give the same."""
import numpy as np
import pytest

from eikonalsolvers import Context, ExtraParams, Grid2DCart, Grid3DCart, api

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


# grids of a 64th of a slot, of no fraction of it, just under and over it
@pytest.mark.parametrize("n,nsrc", [((32, 32), 600), ((17, 13), 3000), ((12, 11, 10), 500), ((255, 257), 9), ((257, 256), 9)])
def test_many_small_grids(monkeypatch, n, nsrc):
    cls = Grid3DCart if len(n) == 3 else Grid2DCart
    grd = cls(hgrid=0.1, cooinit=(0.0,) * len(n), grsize=n)
    rng = np.random.default_rng(nsrc)
    vel = 2.0 + 0.2 * rng.random(n)
    last = 0.1 * (np.array(n) - 1.0)
    cs = rng.uniform(0.1 * last, 0.9 * last, (nsrc, len(n)))
    rec = [rng.uniform(0.05 * last, 0.95 * last, (1, len(n))) for _ in range(nsrc)]
    ep = ExtraParams(refinearoundsrc=False)
    ctx = Context(0)
    try:
        mid = ctx.upload(vel, grd)
        # the first results by plain copies, the later ones through the ring
        rows = [ctx.traveltime(mid, grd, cs, rec, returntt=True, extraparams=ep)[1] for _ in range(3)]
        assert 8 * rows[0][0].size * nsrc >= api.ROWS_MIN_BYTES
        monkeypatch.setattr(api, "ROWS_MIN_BYTES", 1 << 62)  # column-major, put in order by NumPy
        cols = ctx.traveltime(mid, grd, cs, rec, returntt=True, extraparams=ep)[1]
    finally:
        ctx.close()
    for r in rows:
        assert all(np.array_equal(a, b) for a, b in zip(r, cols))
