"""Refined windows whose stop is tied with nodes that are not coarse-coincident are not replayed
(constant and laterally uniform velocities, source off the nodes): traveltimes, gradients and
warnings are those of the exact heap replay; with a coarse-coincident node in the tie they still are."""
import numpy as np
import pytest

from eikonalsolvers import Context, ExtraParams, Grid2DCart, Grid3DCart

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [(61, 47), (30, 31, 29)], ids=["2D", "3D"])
@pytest.mark.parametrize("model", ["constant", "layered"])
@pytest.mark.parametrize("at", ["off", "cell", "node", "border"])
def test_tied_stop_equals_the_replay(ctx, n, model, at):
    nd = len(n)
    cls = Grid3DCart if nd == 3 else Grid2DCart
    grd = cls(hgrid=0.1, cooinit=(0.0,) * nd, grsize=n)
    vel = np.ones(n) if model == "constant" else 1.0 + np.broadcast_to(0.02 * np.arange(n[-1]), n)
    mid = 0.1 * np.floor(np.array(n) / 2.0)
    cs = np.stack([{"off": mid + 0.1 * np.array([0.31, 0.37, 0.43][:nd]), "cell": mid + 0.05, "node": mid,
                    "border": np.where(np.arange(nd) == 0, 0.043, mid + 0.013)}[at] + 0.1 * k for k in range(2)])
    rec = [0.1 * (np.array(n) - 1.0) * np.array([[0.1] * nd, [0.8] * nd, [0.5] * nd]) + 0.02 for _ in range(2)]
    obs, std = [np.full(3, 1.0)] * 2, [np.full(3, 0.1)] * 2
    mod = ctx.upload(vel, grd)
    out, warn, replays = [], [], []
    for mode in (1, 0):
        ctx.set_param("fine_replay", mode)
        picks, tts = ctx.traveltime(mod, grd, cs, rec, returntt=True, extraparams=ExtraParams())
        warn.append(ctx.last_stats.warn_mask)
        replays.append(ctx.last_stats.fine_replays)
        gv, gs, misf = ctx.gradient(mod, grd, cs, rec, obs, std, "gradvelandsrcloc", ExtraParams())
        out.append([*picks, *tts, gv, gs, np.array(misf)])
    ctx.set_param("fine_replay", 0)
    ctx.release(mod)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert warn[0] == warn[1]
    if at == "off":
        assert replays[1] == 0
