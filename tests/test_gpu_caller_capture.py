"""Stream capture by the caller.  A step captured with timestep() is replayed
on a state uploaded in between, which has other cells past phi = 0 than the one
the batch held at the capture; run() is not captured (it launches a graph of its
own, which CUDA does not take into a capture) and leaves the capture as it was."""
import os

import numpy as np
import pytest
import torch

import disco_b200 as db
from disco_b200.workloads import write_par

pytestmark = pytest.mark.gpu

DISKS = [("c0_kepler2d", {"Num_R": 9}),
         ("c1_mhd3d", {"Num_R": 6, "Num_Z": 4, "Constrained_Transport": 0}),
         ("c1_mhd3d", {"Num_R": 6, "Num_Z": 4, "Constrained_Transport": 1})]


def make_disk(base, over):
    p = write_par(over, base=base)
    try:
        return db.Disk.from_files(p, os.path.join(db.TEMPLATES, base + ".in"))
    finally:
        os.unlink(p)


def first_cells(disk, piph):
    """Per annulus the first cell of quadrant I after one of quadrant IV (faces_alt.c:57-79)."""
    out, o = [], 0
    for n in disk.Np:
        phi = piph[o:o + n] * (2 * np.pi / disk.params.phimax)
        q1 = (np.sin(phi) > 0) & (np.cos(phi) > 0)
        q4 = (np.sin(phi) < 0) & (np.cos(phi) > 0)
        i4 = int(np.argmax(q4)) if q4.any() else n
        later = np.flatnonzero(q1[i4 + 1:])
        out.append(i4 + 1 + int(later[0]) if len(later) else 0)
        o += n
    return np.array(out)


def moved_on(b, disk):
    """Run b from its start until the first cells are others than after one step; that early state."""
    b.run(1)
    early = b.get_cells()
    for _ in range(60):
        b.run(5)
        if np.any(first_cells(disk, b.get_cells()["piph"]) != first_cells(disk, early["piph"])):
            return early
    raise AssertionError("the first cells did not change")


def same(a, b):
    for key in a:
        assert np.array_equal(a[key], b[key], equal_nan=True), key


@pytest.mark.parametrize("state", ["kept", "uploaded", "no graph"])
@pytest.mark.parametrize("base,over", DISKS)
def test_replay_after_upload(base, over, state):
    d = make_disk(base, over)
    b, fresh = db.Batch([d]), db.Batch([d])
    s = torch.cuda.Stream()
    b.set_stream(s.cuda_stream)
    if state == "no graph":
        early = b.get_cells()
    else:
        early = moved_on(b, d)
        if state == "uploaded":
            b.set_cells(**b.get_cells())
    b.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        for n in (1, 2):
            with pytest.raises(db.DiscoError):
                b.run(n)
        b.timestep()
    for x in (b, fresh):
        x.set_cells(**early)
        x.mindt()
    for _ in range(2):
        with torch.cuda.stream(s):
            g.replay()
        fresh.timestep()
    s.synchronize()
    same(fresh.get_cells(), b.get_cells())
    b.run(2)                       # the batch's own graph, on the lists the replay left
    for _ in range(2):
        fresh.timestep()
    same(fresh.get_cells(), b.get_cells())
