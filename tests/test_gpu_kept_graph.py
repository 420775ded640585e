"""A batch that holds the graph of its step takes a state whose first cells
past phi = 0 are others than the kept ones, and runs on: the same bits as a
batch that never held a list, for every way of putting a state in."""
import pytest

import disco_b200 as db
from test_gpu_caller_capture import DISKS, first_cells, make_disk, moved_on, same

pytestmark = pytest.mark.gpu


def _put(b, d, how, st):
    if how == "set_cells":
        b.set_cells(**st)
        b.mindt()
    elif how == "restart_cells":
        b.restart_cells(st["prim"], st["piph"], st.get("Phi"))
    else:                          # the initial state on these positions
        b.set_cells(None, None, st["piph"], st["dphi"], st["wiph"])
        db._check(db.library().disco_batch_setup_cells(b.h), "disco_batch_setup_cells")


@pytest.mark.parametrize("how", ["set_cells", "restart_cells", "setup_cells"])
@pytest.mark.parametrize("prec", [db.PREC_FP64, db.PREC_MIXED])
@pytest.mark.parametrize("base,over", DISKS)
def test_run_after_upload(base, over, prec, how):
    d = make_disk(base, over)
    b, fresh = db.Batch([d], precision=prec), db.Batch([d], precision=prec)
    early = moved_on(b, d)
    assert (first_cells(d, b.get_cells()["piph"]) != first_cells(d, early["piph"])).any()
    for x in (b, fresh):
        _put(x, d, how, early)
    for n in (1, 3):
        b.run(n)
        for _ in range(n):
            fresh.timestep()
        same(fresh.get_cells(), b.get_cells())


@pytest.mark.parametrize("base,over", DISKS)
def test_one_step_after_each_upload(base, over):
    """The step after an upload is launched the first time and a graph of its own from then on."""
    d = make_disk(base, over)
    b, fresh = db.Batch([d]), db.Batch([d])
    states = [moved_on(b, d)]
    states += [b.get_cells(), states[0]]
    for n in (1, 2, 1, 3):
        for st in states:
            fresh.set_cells(**st)
            b.set_cells(**st)
            assert b.mindt() == fresh.mindt()
            b.run(n)
            for _ in range(n):
                fresh.timestep()
            same(fresh.get_cells(), b.get_cells())
