"""The forward solve by bricks (8x8x8 or 4x4x4 nodes in 3D, 16x16 or 8x8 in 2D) on grids at and around whole
bricks: smaller than one brick, one node over, ragged in every axis, with and without the
refined start-up, as separate launches and in one. Cartesian grids against the oracle bit for bit;
spherical ones bit for bit between the brick sizes and launches, and within 1e-11 of the oracle (their
source box takes sines and cosines, which the host and the GPU may round differently by an ulp
or two); and the gradient with either brick size, which must not depend on it."""
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
    yield c
    c.close()


@pytest.mark.parametrize("size", [1.0, 2.0], ids=["small", "large"])
@pytest.mark.parametrize("refine", [True, False], ids=["refined", "plain"])
@pytest.mark.parametrize("sphere", [False, True], ids=["cart", "sphere"])
@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
def test_bricks_on_ragged_grids(ctx, n, sphere, refine, size):
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
    out = []
    try:
        for bricks, fused in ((size, 0.0), (size, 2.0), (3.0 - size, 0.0)):
            ctx.set_param("brick_size", bricks)
            ctx.set_param("cluster_solve", fused)
            out.append(ctx.traveltime(mid, grd, cs, rec, returntt=True, extraparams=ep))
    finally:
        ctx.set_param("brick_size", 0.0)
        ctx.set_param("cluster_solve", 1.0)
        ctx.release(mid)
    op, ott = O.eiktraveltime(vel, grd, cs, rec, returntt=True, extraparams=ep)
    for s in range(2):
        for picks, tt in out[1:]:
            assert np.array_equal(tt[s], out[0][1][s]) and np.array_equal(picks[s], out[0][0][s])
        picks, tt = out[0]
        if sphere:
            np.testing.assert_allclose(tt[s], ott[s], rtol=1e-11, atol=0.0)
            np.testing.assert_allclose(picks[s], op[s], rtol=1e-11, atol=0.0)
        else:
            assert np.array_equal(tt[s], ott[s]) and np.array_equal(picks[s], op[s])


@pytest.mark.parametrize("n", [(17, 33), (50, 31), (9, 17, 8), (20, 21, 26)], ids=lambda n: "x".join(map(str, n)))
def test_gradient_does_not_depend_on_the_brick_size(ctx, n):
    rng = np.random.default_rng(sum(n))
    nd = len(n)
    grd = (Grid3DCart if nd == 3 else Grid2DCart)(hgrid=0.5, cooinit=(0.0,) * nd, grsize=n)
    vel = np.ascontiguousarray(3.0 * np.exp(0.25 * rng.standard_normal(n)))
    ext = [0.5 * (m - 1) for m in n]
    cs = np.array([[e * rng.uniform(0.05, 0.95) for e in ext] for _ in range(3)])
    rec = [np.array([[e * rng.uniform(0.0, 1.0) for e in ext] for _ in range(37)]) for _ in range(3)]
    po = [np.linalg.norm(r - c, axis=1) / 3.0 for r, c in zip(rec, cs)]
    so = [np.full(37, 0.1) for _ in range(3)]
    mid = ctx.upload(vel, grd)
    try:
        out = []
        for size in (1.0, 2.0):
            ctx.set_param("brick_size", size)
            out.append(ctx.gradient(mid, grd, cs, rec, po, so, "gradvelandsrcloc"))
    finally:
        ctx.set_param("brick_size", 0.0)
        ctx.release(mid)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    ov, os_, om = O.eikgradient(vel, grd, cs, rec, po, so, "gradvelandsrcloc", extraparams=ExtraParams())
    assert np.linalg.norm(out[0][0] - ov) <= 1e-10 * np.linalg.norm(ov)
    assert np.linalg.norm(out[0][1] - os_) <= 1e-10 * np.linalg.norm(os_)
