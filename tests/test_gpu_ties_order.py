"""Refined windows with a tied stop beside sharp layers. Where non-causal acceptances follow one another (keys of
depth 2 and more) the window is replayed, as its traveltimes depend on the heap's order; where they do not, it is
not, and the warning of a negative discriminant comes from the fixed point: traveltimes, gradients and
warnings are the replay's either way."""
import numpy as np
import pytest

from eikonalsolvers import Context, ExtraParams, Grid2DCart, Grid3DCart

pytestmark = pytest.mark.gpu

NEGATIVE_DISCRIMINANT = 1


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def _column(first, last, velocity):
    col = np.ones(30)
    col[first:last] = velocity
    return col


# dimension, velocities along the last axis, source in its cell, replayed, warns
CASES = {
    "2D-chain": (2, _column(13, 14, 20.0), (0.2, 0.2), 1, True),
    "3D-chain": (3, _column(16, 30, 20.0), (0.31, 0.37, 0.43), 1, True),
    "3D-chain-sheet": (3, _column(16, 17, 20.0), (0.31, 0.37, 0.43), 1, True),
    "2D-warns": (2, _column(15, 30, 10.0), (0.35, 0.35), 0, True),
    "2D-warns-sheet": (2, _column(15, 16, 10.0), (0.35, 0.35), 0, True),
    "2D-warns-slow": (2, _column(14, 15, 0.1), (0.35, 0.35), 0, True),
    "2D-clear": (2, _column(15, 30, 10.0), (0.2, 0.2), 0, False),
    "3D-clear": (3, _column(15, 30, 10.0), (0.2, 0.2, 0.45), 0, False),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tied_windows_beside_layers(ctx, name):
    nd, col, at, replayed, warns = CASES[name]
    n = (30,) * nd
    grd = (Grid3DCart if nd == 3 else Grid2DCart)(hgrid=0.1, cooinit=(0.0,) * nd, grsize=n)
    cs = 1.4 + 0.1 * np.array([at])
    rec = [0.1 * 29 * np.array([[0.1] * nd, [0.8] * nd, [0.5] * nd]) + 0.02]
    obs, std = [np.full(3, 1.0)], [np.full(3, 0.1)]
    mid = ctx.upload(np.broadcast_to(col, n).copy(), grd)
    out, warn, replays = [], [], []
    try:
        for mode in (1.0, 0.0):
            ctx.set_param("fine_replay", mode)
            picks, tts = ctx.traveltime(mid, grd, cs, rec, returntt=True, extraparams=ExtraParams())
            warn.append(ctx.last_stats.warn_mask)
            replays.append(ctx.last_stats.fine_replays)
            gv, gs, misf = ctx.gradient(mid, grd, cs, rec, obs, std, "gradvelandsrcloc", ExtraParams())
            out.append([*picks, *tts, gv, gs, np.array(misf)])
    finally:
        ctx.set_param("fine_replay", 0.0)
        ctx.release(mid)
    assert replays[1] == replayed
    assert warn[0] == warn[1] and bool(warn[1] & NEGATIVE_DISCRIMINANT) == warns
    for a, b in zip(*out):
        assert np.array_equal(a, b)
