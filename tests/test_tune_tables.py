"""Tables of tuned widths across solvers and brick sizes: entries kept from another solver are not applied and stay
in the file; a width tuned with one brick size is not used with the other."""
import json

from eikonalsolvers import Grid2DCart, Grid3DCart
from eikonalsolvers.tune import SOLVER, Tuner, small_bricks, workload_key


class Fake:
    def __init__(self):
        self.params = {}

    def set_param(self, name, value):
        self.params[name] = value


def _grid(n):
    return (Grid3DCart if len(n) == 3 else Grid2DCart)(hgrid=1.0, cooinit=(0.0,) * len(n), grsize=n)


def test_entries_of_another_solver_are_not_applied(tmp_path):
    path = str(tmp_path / "tune.json")
    grd = _grid((300, 220))
    key = workload_key(grd, 4)
    old = {"round_gate": 2.0, "ctas_per_sm": 3, "ms": 9.9, "timings": [[2.0, 3, 9.9]]}
    json.dump({key: old, "Grid2DCart:n131072:s4:r1": old}, open(path, "w"))
    t = Tuner(path=path, shipped=None)
    ctx = Fake()
    assert t.apply_known(ctx, grd, 4) is None and ctx.params == {}
    t.table[key] = dict(old, round_gate=64.0, solver=SOLVER)
    t._save()
    kept = json.load(open(path))
    assert kept["Grid2DCart:n131072:s4:r1"] == old and kept[key]["round_gate"] == 64.0
    assert Tuner(path=path, shipped=None).apply_known(ctx, grd, 4)["round_gate"] == 64.0


def test_brick_sizes_do_not_share_an_entry():
    # one class by powers of two, on both sides of the library's choice of bricks
    for a, b, nsrc in (((1024, 640), (1024, 1024), 64), ((118, 119, 120), (128, 128, 128), 12)):
        assert small_bricks(_grid(a), nsrc) and not small_bricks(_grid(b), nsrc)
        ka, kb = workload_key(_grid(a), nsrc), workload_key(_grid(b), nsrc)
        assert ka != kb and ka.rsplit(":", 1)[0] == kb.rsplit(":", 1)[0]


def test_shipped_entries_are_this_solvers():
    t = Tuner(path="")
    assert t.base and all(e["solver"] == SOLVER for e in t.base.values())
