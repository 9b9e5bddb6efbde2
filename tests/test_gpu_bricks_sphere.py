"""Gradients on spherical grids of several radial bricks, ragged in every axis: the same with either brick size (the
adjoint keeps a brick's spherical coefficients in unread parts of its cube), and the oracle's. And the size up
to which a 2D solve is one launch: 2^20 node-sources, the same results on both sides."""
import numpy as np
import pytest

import eikoracle as O
from eikonalsolvers import Context, ExtraParams, Grid2DCart, Grid2DSphere, Grid3DSphere

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("refine", [True, False], ids=["refined", "plain"])
@pytest.mark.parametrize("n", [(33, 47), (18, 17), (20, 21, 26), (9, 17, 8), (27, 12, 19)], ids=lambda n: "x".join(map(str, n)))
def test_spherical_gradient_does_not_depend_on_the_brick_size(ctx, n, refine):
    rng = np.random.default_rng(sum(n) + refine)
    nd = len(n)
    co, sp = np.array((5800.0, 80.0, 80.0)[:nd]), np.array((4.0, 0.05, 0.04)[:nd])
    cls = Grid3DSphere if nd == 3 else Grid2DSphere
    kw = dict(zip(("Δr", "Δθ", "Δφ"), sp))
    grd = cls(**kw, cooinit=tuple(co), grsize=n)
    vel = np.ascontiguousarray(5.0 * np.exp(0.2 * rng.standard_normal(n)))
    ext = sp * (np.array(n) - 1)
    cs = co + ext * rng.uniform(0.05, 0.95, (3, nd))
    rec = [co + ext * rng.uniform(0.0, 1.0, (37, nd)) for _ in range(3)]
    ep = ExtraParams(refinearoundsrc=refine)
    obs = O.eiktraveltime(vel, grd, cs, rec, extraparams=ep)
    po, so = [1.05 * p for p in obs], [np.full(37, 0.1)] * 3
    mid = ctx.upload(vel, grd)
    try:
        out = []
        for size in (1.0, 2.0):
            ctx.set_param("brick_size", size)
            out.append(ctx.gradient(mid, grd, cs, rec, po, so, "gradvel", extraparams=ep))
    finally:
        ctx.set_param("brick_size", 0.0)
        ctx.release(mid)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    ov, om = O.eikgradient(vel, grd, cs, rec, po, so, "gradvel", extraparams=ep)
    # as for the spherical traveltimes: host and GPU may round a source box's sines and cosines differently by an
    # ulp or two, which the adjoint's sums of differences enlarge
    assert np.linalg.norm(out[0][0] - ov) <= 1e-8 * np.linalg.norm(ov)
    assert abs(out[0][1] - om) <= 1e-8 * abs(om)


def test_fused_up_to_2_20_node_sources(ctx):
    rec = [np.array([[10.3, 20.4], [500.5, 700.25]])]
    cs = np.array([[333.3, 444.4]])
    ep = ExtraParams(refinearoundsrc=False)
    for n, fused in (((1024, 1024), True), ((1024, 1025), False)):
        grd = Grid2DCart(hgrid=1.0, cooinit=(0.0, 0.0), grsize=n)
        vel = 3.0 * np.exp(0.1 * np.random.default_rng(n[1]).standard_normal(n))
        mid = ctx.upload(vel, grd)
        out, launches = [], []
        try:
            for mode in (1.0, 0.0):
                ctx.set_param("cluster_solve", mode)
                out.append(ctx.traveltime(mid, grd, cs, rec, extraparams=ep)[0])
                launches.append(ctx.last_stats.launches)
        finally:
            ctx.set_param("cluster_solve", 1.0)
            ctx.release(mid)
        assert np.array_equal(*out)
        # counters and the solve against counters, reset, seeds, solve and store
        assert launches[1] - launches[0] == (3 if fused else 0)
