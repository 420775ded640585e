"""timestep(dt) takes its dt at the call: a capture would step with that dt at
every replay, so it is refused there, and the batch goes on as before."""
import numpy as np
import pytest
import torch

import disco_b200 as db
from test_gpu_caller_capture import make_disk, same

pytestmark = pytest.mark.gpu


def test_timestep_with_dt_is_not_captured():
    d = make_disk("c0_kepler2d", {"Num_R": 5})
    b, other = db.Batch([d]), db.Batch([d])
    s = torch.cuda.Stream()
    b.set_stream(s.cuda_stream)
    dt = b.mindt()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        with pytest.raises(db.DiscoError):
            b.timestep(dt)
        b.timestep()               # the step with the device's own dt can be captured
    b.timestep(dt)
    other.timestep(np.array(other.mindt()))
    same(other.get_cells(), b.get_cells())
