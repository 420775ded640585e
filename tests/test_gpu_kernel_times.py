"""Every row of kernel_times is a launch of its own with its device time: on
annuli of many cells whose first cell lies just past phi = 0, the search for
the next such cell walks the annulus to its end, and its row shows it."""
import numpy as np
import pytest

import disco_b200 as db
from test_gpu_caller_capture import make_disk

pytestmark = pytest.mark.gpu


def test_search_for_first_cells_has_its_time():
    d = make_disk("c0_kepler2d", {"Num_R": 4, "aspect": 0.001, "Max_Aspect_Short": 1e5, "Max_Aspect_Long": 1e5})
    assert d.Np.min() > 4000                   # 125 rounds of 32 cells, a double sincos in each
    b = db.Batch([d])
    st = b.get_cells()
    st["piph"] = np.concatenate([(np.arange(n) + 0.5) * (d.params.phimax / n) for n in d.Np])
    ms = []
    for _ in range(5):
        b.set_cells(**st)
        b.mindt()
        rows = [t for name, t in b.kernel_times() if name == "k_I0"]
        assert len(rows) == 2
        ms.append(rows[0])                     # nothing kept after an upload
    # 125 dependent rounds of a load (over 100 ns each on any GPU) against an
    # interval without a launch (about 2 us)
    assert np.median(ms) > 0.010


@pytest.mark.parametrize("base,over,rows", [
    ("c0_kepler2d", {"Num_R": 9}, 2 * 6 + 1),          # begin, faces, grad, flux, update, c2p; step end
    # and the zero-gradient copies in r and in z; the diagnostics' sums after the last of them
    ("c1_mhd3d", {"Num_R": 6, "Num_Z": 4}, 2 * 8 + 2)])
def test_one_row_per_launch(base, over, rows):
    b = db.Batch([make_disk(base, dict(over, Constrained_Transport=0))])
    b.run(2)
    kt = b.kernel_times()
    assert sum(name != "k_I0" for name, _ in kt) == rows
    assert all(t > 0 for _, t in kt)
