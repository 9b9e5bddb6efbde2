"""Results that cross to pageable memory by chunks, row-major grids and models reordered on the
device: the same bytes as the plain column-major calls give, at sizes around the chunk."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from eikonalsolvers import Context
    c = Context(0)
    yield c
    c.close()


def _workload(n, nsrc):
    from eikonalsolvers import Grid2DCart, Grid3DCart
    cls = Grid3DCart if len(n) == 3 else Grid2DCart
    grd = cls(hgrid=0.1, cooinit=(0.0,) * len(n), grsize=n)
    rng = np.random.default_rng(len(n) * 1000 + n[0])
    vel = 2.0 + 0.2 * rng.random(n) + np.linspace(0.0, 1.0, n[-1])
    last = 0.1 * (np.array(n) - 1.0)
    cs = rng.uniform(0.3 * last, 0.7 * last, (nsrc, len(n)))
    rec = [rng.uniform(0.05 * last, 0.95 * last, (4, len(n))) for _ in range(nsrc)]
    return grd, vel, cs, rec


# grids of less than the row-major path's least size, of it, with a ragged last chunk of 1 MB
# and 2 MB, and several chunks a grid
@pytest.mark.parametrize("n,nsrc", [((64, 50), 3), ((512, 512), 2), ((61, 73, 59), 3), ((1031, 777), 1), ((40, 41, 43), 9)])
def test_row_major_grids_are_the_column_major_ones(ctx, n, nsrc):
    from eikonalsolvers import _lib
    grd, vel, cs, rec = _workload(n, nsrc)
    mid = ctx.upload(vel, grd)
    picks, tts = ctx.traveltime(mid, grd, cs, rec, returntt=True)
    N = int(np.prod(n))
    off = np.arange(0, 4 * nsrc + 1, 4, dtype=np.int64)
    pk, flat = np.zeros(4 * nsrc), np.zeros(nsrc * N)
    ep, st = _lib.extra_struct(None), _lib.eik_stats()
    _lib.check(ctx.L.eik_traveltime(ctx.h, C.c_int64(mid), nsrc, _lib.ptr(np.ascontiguousarray(cs)), _lib.ptr(off),
                                    _lib.ptr(np.concatenate(rec)), C.byref(ep), _lib.ptr(pk), _lib.ptr(flat),
                                    C.byref(st)), ctx.h)
    for s in range(nsrc):
        assert tts[s].shape == tuple(n) and tts[s].flags.c_contiguous and tts[s].flags.owndata
        assert np.array_equal(tts[s], flat[s * N:(s + 1) * N].reshape(n, order="F"))
        assert np.array_equal(picks[s], pk[4 * s:4 * s + 4])
    ctx.release(mid)


@pytest.mark.parametrize("n", [(64, 50), (61, 73, 59)])
def test_models_of_either_order_are_the_same(ctx, n):
    grd, vel, cs, rec = _workload(n, 2)
    out = []
    for v in (vel, np.asfortranarray(vel), np.repeat(vel, 2, axis=0)[::2]):
        mid = ctx.upload(v, grd)
        out.append(ctx.traveltime(mid, grd, cs, rec))
        ctx.release(mid)
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], o))


# below and above the least size of the chunked copy, with a ragged last chunk
@pytest.mark.parametrize("n", [(61, 73, 59), (101, 103, 107)])
def test_gradient_to_pageable_and_to_pinned_memory(ctx, n):
    import torch
    from eikonalsolvers import _lib
    grd, vel, cs, rec = _workload(n, 1)
    mid = ctx.upload(vel, grd)
    obs, std = [np.full(4, 1.0)], [np.full(4, 0.1)]
    grad, _ = ctx.gradient(mid, grd, cs, rec, obs, std, "gradvel")
    N = int(np.prod(n))
    pinned = torch.zeros(N, dtype=torch.float64, pin_memory=True)
    off = np.array([0, 4], dtype=np.int64)
    ep, st, misf = _lib.extra_struct(None), _lib.eik_stats(), np.zeros(1)
    _lib.check(ctx.L.eik_gradient(ctx.h, C.c_int64(mid), 1, _lib.ptr(np.ascontiguousarray(cs)), _lib.ptr(off),
                                  _lib.ptr(rec[0]), _lib.ptr(obs[0]), _lib.ptr(std[0]), 1, C.byref(ep),
                                  C.c_void_p(pinned.data_ptr()), None, _lib.ptr(misf), C.byref(st)), ctx.h)
    assert np.array_equal(grad, pinned.numpy().reshape(n, order="F"))
    ctx.release(mid)
