"""A batch that does not fit the device's free memory is an error of
disco_batch_create, before any kernel is launched, and leaves the memory it
had taken and the context as they were."""
import pytest
import torch

import disco_b200 as db
from test_gpu_caller_capture import make_disk

pytestmark = pytest.mark.gpu


def test_batch_larger_than_free_memory():
    big = make_disk("c1_mhd3d", {"Num_R": 80, "Num_Z": 60, "Constrained_Transport": 1})
    small = make_disk("c0_kepler2d", {"Num_R": 5})
    want = db.Batch([small])                   # the library and its context are loaded
    want.run(2)
    assert big.ncell * 1200 > 2**30            # cons, RKcons, prims, slopes, fluxes alone
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - 2**30, dtype=torch.uint8, device="cuda")
    left = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        with pytest.raises(db.DiscoError):
            db.Batch([big], setup=False)
        assert left - torch.cuda.mem_get_info()[0] < 2**26
    del fill
    torch.cuda.empty_cache()
    b = db.Batch([small])
    b.run(2)
    assert (b.get_cells()["prim"] == want.get_cells()["prim"]).all()
