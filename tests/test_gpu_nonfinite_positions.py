"""Cell positions that are not finite, in the first state a batch gets or in a
later one: every face run and every edge rank that the kernels follow lies
within its track and line, so the step ends, with an error status where a
position is infinite (a NaN fails every comparison, the phi wraps' too, and may
pass unnoticed, as in the reference).  The context stays usable and a clean
state steps to the bits of a batch that never saw them."""
import numpy as np
import pytest

import disco_b200 as db
from test_gpu_caller_capture import DISKS, make_disk, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("base,over", DISKS)
def test_non_finite_positions(base, over, first, bad):
    d = make_disk(base, over)
    want = db.Batch([d])
    clean = want.get_cells()
    b = db.Batch([d], setup=False) if first else db.Batch([d])
    if not first:
        b.run(2)
    rng = np.random.default_rng(5)
    piph = clean["piph"].copy()
    piph[rng.choice(d.ncell, max(3, d.ncell // 50), replace=False)] = bad
    b.set_cells(**dict(clean, piph=piph))
    b.timestep(want.mindt())
    assert b.last_error() in ((4, 5, 8) if np.isinf(bad) else (0, 4, 5, 8))
    dt = want.mindt()
    b.set_cells(**clean)
    want.set_cells(**clean)
    for x in (b, want):
        for _ in range(2):
            x.timestep(dt)
    assert b.last_error() == 0
    same(want.get_cells(), b.get_cells())
