"""Where the batch knows its face lists to be those of the current positions,
the first substep does not look for them again.  A state uploaded in between,
and a step that the caller captured and replays, must not rely on that: the
same bits as a batch that never kept a list."""
import os

import numpy as np
import pytest
import torch

import disco_b200 as db
from disco_b200.workloads import write_par

pytestmark = pytest.mark.gpu


def _disk(base, **over):
    p = write_par(over, base=base)
    d = db.Disk.from_files(p, os.path.join(db.TEMPLATES, base + ".in"))
    os.unlink(p)
    return d


DISKS = [("c0_kepler2d", {"Num_R": 9}), ("c1_mhd3d", {"Num_R": 6, "Num_Z": 4})]


def _same(a, b):
    for key in a:
        assert np.array_equal(a[key], b[key], equal_nan=True), key


@pytest.mark.parametrize("base,over", DISKS)
def test_upload_between_runs(base, over):
    d = _disk(base, **over)
    b = db.Batch([d])
    b.run(1)
    early = b.get_cells()
    b.run(20)                                  # the positions of `early` are gone
    fresh = db.Batch([d])
    got = []
    for x in (b, fresh):
        x.set_cells(**early)
        for _ in range(3):
            x.timestep(x.mindt())
        got.append(x.get_cells())
    _same(got[0], got[1])


@pytest.mark.parametrize("base,over", DISKS)
def test_captured_step(base, over):
    d = _disk(base, **over)
    want = db.Batch([d])
    want.run(4)
    b = db.Batch([d])
    s = torch.cuda.Stream()
    b.set_stream(s.cuda_stream)
    b.run(2)
    b.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        b.timestep()
    with torch.cuda.stream(s):
        g.replay()
        g.replay()
    s.synchronize()
    _same(want.get_cells(), b.get_cells())
