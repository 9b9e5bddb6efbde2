"""The forward solve by bricks, emulated on the host (brick_schedule_harness.cpp: the visits and rounds of
brick.cuh and coarse.cu restated around the product's order rule, stencil.cuh compiled for the host), reaches the
oracle's heap-FMM traveltimes bit for bit with either brick size, at any round width and with visits cut
off after a single scan; and with the fast form of the rule it ends where the general rule does."""
import os
import shutil
import struct
import subprocess

import numpy as np
import pytest

import eikoracle as O
import refcases as RC
from blockmodels import block_model, contrast_model
from eikonalsolvers import ExtraParams, Grid3DCart
from eikonalsolvers import configs as CF

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "eikonalsolvers.jl_b200", "csrc")
ROUNDS = 1 << 16


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("bricks")
    exe = str(d / "harness")
    cmd = ["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
           os.path.join(HERE, "brick_schedule_harness.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return exe, d


def _emulate(harness, vel, grd, src, gate, small, scans=0, general=0):
    """One source without refined start-up: (emulated traveltimes, the oracle's, counters)."""
    exe, d = harness
    dbg = O.forward_debug(vel, grd, np.asarray(src, dtype=np.float64), extraparams=ExtraParams(refinearoundsrc=False))
    tt = dbg["tt"].ravel(order="F")
    seeds = np.ascontiguousarray(dbg["srcpts"], dtype=np.int64)
    slow = 1.0 / np.asarray(vel, dtype=np.float64).ravel(order="F")  # as the product's slowness kernel
    n = list(grd.grsize) + [1] * (3 - grd.ndim)
    fin, fout = str(d / "in.bin"), str(d / "out.bin")
    with open(fin, "wb") as f:
        f.write(struct.pack("<4i2d4iq", grd.ndim, *n, grd.hgrid, gate, small, scans, general, ROUNDS, seeds.size))
        f.write(slow.tobytes())
        f.write(seeds.tobytes())
        f.write(np.ascontiguousarray(tt[seeds]).tobytes())
    subprocess.run([exe, fin, fout], check=True)
    out = np.fromfile(fout, dtype=np.float64, count=tt.size)
    st = np.fromfile(fout, dtype=np.int64, offset=8 * tt.size)
    return out, tt, dict(zip(("rounds", "evals", "left", "unsettled", "tied"), (int(x) for x in st)))


def _check(out, tt, st):
    assert int((out != tt).sum()) == 0
    assert st["rounds"] < ROUNDS and st["unsettled"] == 0


# round width, small bricks, scans of a visit (0: the product's), general rule only
SCHEDULES = [(8.0, 1, 0, 0), (6.0, 0, 0, 0), (1.0, 1, 1, 0), (64.0, 0, 1, 0), (64.0, 1, 200, 0), (16.0, 0, 0, 1)]


@pytest.mark.parametrize("case", RC.all_forward_cases(), ids=lambda c: c["name"])
def test_reference_cases(harness, case):
    src = np.atleast_2d(case["coordsrc"])[0]
    for s in SCHEDULES:
        _check(*_emulate(harness, case["vel"], case["grd"], src, *s))


_WORKLOADS = {
    "300x220": lambda: CF.cfg1(),
    "32cubed": lambda: CF.cfg3(scale=0.125, nsrc=2, nrec_side=3),
    "128x80_random_field": lambda: CF.cfg2(scale=0.125, nsrc=2),
}


@pytest.mark.parametrize("which", sorted(_WORKLOADS))
def test_seeded_workloads(harness, which):
    w = _WORKLOADS[which]()
    for src in w.coordsrc[:2]:
        for s in SCHEDULES:
            _check(*_emulate(harness, w.vel, w.grd, src, *s))


@pytest.mark.parametrize("seed", [55, 78, 106, 256, 316, 404])
def test_block_models_with_tied_keys(harness, seed):
    """Blocks of round velocities whose solve meets a special key with level equal to traveltime."""
    vel, src = block_model((40, 40, 40), seed)
    grd = Grid3DCart(hgrid=1.0, cooinit=(0.0, 0.0, 0.0), grsize=(40, 40, 40))
    for s in SCHEDULES:
        out, tt, st = _emulate(harness, vel, grd, src, *s)
        _check(out, tt, st)
        assert st["tied"] > 0


@pytest.mark.parametrize("kind,contrast,seed", [("blocks", 40.0, 4), ("blocks", 100.0, 4), ("noise", 100.0, 4),
                                                ("noise", 1000.0, 4), ("smooth", 1000.0, 4), ("lens", 40.0, 4),
                                                ("lens", 100.0, 4)])
def test_high_contrast_models_settle(harness, kind, contrast, seed):
    """Nodes of a slow region wait many round widths for the front, more of them apart than a visit has scans:
    evaluating them again must not keep a visit from the nodes that can change."""
    n = (24, 24, 24)
    grd = Grid3DCart(hgrid=1.0, cooinit=(0.0, 0.0, 0.0), grsize=n)
    for gate, small in ((6.0, 0), (8.0, 1)):
        out, tt, st = _emulate(harness, contrast_model(kind, n, contrast, seed), grd, (9.01, 9.01, 9.01), gate, small)
        _check(out, tt, st)
        assert st["evals"] < 20 * out.size
