"""A step whose launches the driver refuses has built no face lists: the next
one must not take them as kept.  The refusal here is a launch on the legacy
stream while another stream is being captured."""
import ctypes as C

import pytest

import disco_b200 as db
from test_gpu_caller_capture import make_disk, moved_on, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["run", "timestep"])
def test_refused_step_leaves_no_lists(call):
    rt = C.CDLL("libcudart.so.12")
    d = make_disk("c0_kepler2d", {"Num_R": 9})
    b, fresh = db.Batch([d]), db.Batch([d])
    early = moved_on(b, d)
    for x in (b, fresh):
        x.set_cells(**early)
        x.mindt()
    b.set_stream(1)                            # cudaStreamLegacy
    s, g = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreate(C.byref(s)) == 0
    assert rt.cudaStreamBeginCapture(s, 0) == 0
    try:
        with pytest.raises(db.DiscoError):
            b.run(1) if call == "run" else b.timestep()
    finally:
        rt.cudaStreamEndCapture(s, C.byref(g))
        rt.cudaGetLastError()
        rt.cudaStreamDestroy(s)
    b.set_stream(None)
    same(fresh.get_cells(), b.get_cells())     # nothing of the step ran
    b.run(2)
    for _ in range(2):
        fresh.timestep()
    same(fresh.get_cells(), b.get_cells())
