"""3D models of blocks with round velocities, whose solves meet special keys with level equal to traveltime
(exact ties beside shocks), and models of high velocity contrast, whose slow nodes wait many rounds: with either
brick size the oracle's traveltimes bit for bit."""
import numpy as np
import pytest

import eikoracle as O
from blockmodels import block_model, contrast_model
from eikonalsolvers import Context, ExtraParams, Grid3DCart

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("seed,refine", [(55, False), (78, False), (106, False), (256, False), (316, False), (404, False),
                                         (55, True), (228, True), (316, True)])
def test_tied_keys_on_block_models(ctx, seed, refine):
    vel, src = block_model((40, 40, 40), seed)
    grd = Grid3DCart(hgrid=1.0, cooinit=(0.0, 0.0, 0.0), grsize=(40, 40, 40))
    rec = [np.array([[3.3, 4.4, 5.5], [36.1, 20.2, 11.3]])]
    ep = ExtraParams(refinearoundsrc=refine)
    op, ott = O.eiktraveltime(vel, grd, src[None, :], rec, returntt=True, extraparams=ep)
    mid = ctx.upload(vel, grd)
    try:
        for size in (1.0, 2.0):
            ctx.set_param("brick_size", size)
            picks, tt = ctx.traveltime(mid, grd, src[None, :], rec, returntt=True, extraparams=ep)
            assert np.array_equal(tt[0], ott[0]) and np.array_equal(picks[0], op[0])
    finally:
        ctx.set_param("brick_size", 0.0)
        ctx.release(mid)


@pytest.mark.parametrize("kind,contrast", [("blocks", 40.0), ("blocks", 100.0), ("noise", 100.0), ("noise", 1000.0),
                                           ("smooth", 1000.0), ("lens", 40.0), ("lens", 100.0)])
def test_high_contrast_models_settle(ctx, kind, contrast):
    n = (24, 24, 24)
    vel = contrast_model(kind, n, contrast, 4)
    grd = Grid3DCart(hgrid=1.0, cooinit=(0.0, 0.0, 0.0), grsize=n)
    src, rec = np.array([[9.01, 9.01, 9.01]]), [np.array([[3.3, 4.4, 5.5]])]
    ep = ExtraParams(refinearoundsrc=False)
    op, ott = O.eiktraveltime(vel, grd, src, rec, returntt=True, extraparams=ep)
    mid = ctx.upload(vel, grd)
    try:
        ctx.set_param("max_rounds", 20000.0)  # a few hundred to two thousand in practice
        for size in (1.0, 2.0):
            ctx.set_param("brick_size", size)
            picks, tt = ctx.traveltime(mid, grd, src, rec, returntt=True, extraparams=ep)
            assert np.array_equal(tt[0], ott[0]) and np.array_equal(picks[0], op[0])
    finally:
        ctx.set_param("max_rounds", 0.0)
        ctx.set_param("brick_size", 0.0)
        ctx.release(mid)
