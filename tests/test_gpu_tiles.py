"""The cell and face arrays lie in tiles with the fields of a tile one
after another: whatever cell a disk starts at inside a tile, and wherever the
batch ends, a state comes back as it was set and the disk steps to the same bits
as alone."""
import os

import numpy as np
import pytest

import disco_b200 as db
from disco_b200.workloads import write_par

pytestmark = pytest.mark.gpu

TILE = 32


def _disk(base, **over):
    p = write_par(over, base=base)
    d = db.Disk.from_files(p, os.path.join(db.TEMPLATES, {
        "c0_kepler2d": "c0_kepler2d.in", "c1_mhd2d": "c1_mhd2d.in", "c1_mhd3d": "c1_mhd3d.in",
        "c4_binary3d": "c4_binary3d.in"}[base]))
    os.unlink(p)
    return d


@pytest.mark.parametrize("prec", [db.PREC_FP64, db.PREC_MIXED])
@pytest.mark.parametrize("base,over,lead", [
    ("c0_kepler2d", {"Num_R": 5}, [{"Num_R": n} for n in (3, 4, 6, 9)]),
    ("c1_mhd2d", {"Num_R": 6}, [{"Num_R": n} for n in (5, 8)]),
    ("c1_mhd3d", {"Num_R": 5, "Num_Z": 4}, [{"Num_R": n, "Num_Z": 3} for n in (4, 6)]),
    ("c4_binary3d", {"Num_R": 6, "Num_Z": 4}, [{"Num_R": n, "Num_Z": 3} for n in (5, 8)])])
def test_disk_at_any_offset(base, over, lead, prec):
    x = _disk(base, **over)
    alone = db.Batch([x], precision=prec)
    start = alone.get_cells()
    alone.run(3)
    want = alone.get_cells()
    ends = set()
    for o in lead:
        first = _disk(base, **o)
        b = db.Batch([first, x], precision=prec)
        n0 = int(np.sum(first.Np))
        ends |= {n0 % TILE, b.ncell % TILE}
        got = b.get_cells()
        for key, a in start.items():
            assert np.array_equal(got[key][n0:], a, equal_nan=True), (key, n0)
        b.run(3)
        got = b.get_cells()
        for key, a in want.items():
            assert np.array_equal(got[key][n0:], a, equal_nan=True), (key, n0)
        rng = np.random.default_rng(n0)
        put = dict(got)
        for key in ("prim", "cons", "Phi"):
            if key in put:
                put[key] = rng.standard_normal(put[key].shape).astype(np.float32).astype(np.float64)
        b.set_cells(**put)
        back = b.get_cells()
        for key, a in put.items():
            assert np.array_equal(back[key], a, equal_nan=True), (key, n0)
    assert len(ends) > 1                       # offsets inside a tile
