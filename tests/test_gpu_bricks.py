"""The forward solve by bricks (8x8x8 nodes in 3D, 16x16 in 2D) on grids at and around whole
bricks: smaller than one brick, one node over, ragged in every axis, with and without the
refined start-up. Cartesian grids against the oracle, spherical ones against the cluster solve
(their source box takes sines and cosines, which the host and the GPU may round differently),
both bit for bit."""
import numpy as np
import pytest

import eikoracle as O
from eikonalsolvers import Context, ExtraParams, Grid2DCart, Grid2DSphere, Grid3DCart, Grid3DSphere

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3), (15, 16), (16, 16), (17, 33), (47, 18), (3, 3, 3), (7, 8, 9), (8, 8, 8), (9, 17, 8), (16, 25, 10),
          (5, 40, 24)]


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    c.set_param("cluster_solve", 0.0)
    yield c
    c.close()


@pytest.mark.parametrize("refine", [True, False], ids=["refined", "plain"])
@pytest.mark.parametrize("sphere", [False, True], ids=["cart", "sphere"])
@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
def test_bricks_on_ragged_grids(ctx, n, sphere, refine):
    rng = np.random.default_rng(sum(n) + refine)
    nd = len(n)
    if sphere:
        co = (5800.0, 80.0, 80.0)[:nd]
        sp = (4.0, 0.05, 0.04)[:nd]
        grd = (Grid3DSphere(Δr=sp[0], Δθ=sp[1], Δφ=sp[2], cooinit=co, grsize=n) if nd == 3
               else Grid2DSphere(Δr=sp[0], Δθ=sp[1], cooinit=co, grsize=n))
    else:
        co, sp = (0.0,) * nd, (0.5,) * nd
        grd = Grid3DCart(hgrid=0.5, cooinit=co, grsize=n) if nd == 3 else Grid2DCart(hgrid=0.5, cooinit=co, grsize=n)
    vel = np.ascontiguousarray(3.0 * np.exp(0.25 * rng.standard_normal(n)))
    ext = [sp[d] * (n[d] - 1) for d in range(nd)]
    cs = np.array([[co[d] + ext[d] * rng.uniform(0.05, 0.95) for d in range(nd)] for _ in range(2)])
    rec = [np.array([[co[d] + ext[d] * rng.uniform(0.0, 1.0) for d in range(nd)] for _ in range(4)]) for _ in range(2)]
    ep = ExtraParams(refinearoundsrc=refine)
    mid = ctx.upload(vel, grd)
    try:
        picks, tt = ctx.traveltime(mid, grd, cs, rec, returntt=True, extraparams=ep)
        if sphere:
            ctx.set_param("cluster_solve", 2.0)
            op, ott = ctx.traveltime(mid, grd, cs, rec, returntt=True, extraparams=ep)
            ctx.set_param("cluster_solve", 0.0)
        else:
            op, ott = O.eiktraveltime(vel, grd, cs, rec, returntt=True, extraparams=ep)
    finally:
        ctx.release(mid)
    for s in range(2):
        assert np.array_equal(tt[s], ott[s])
        assert np.array_equal(picks[s], op[s])
