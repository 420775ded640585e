"""The conserved variables of ghost cells take part in the Runge-Kutta average
alone (adjust_RK_cons, misc.c:226-244): (1-RK) c + RK c0 leaves a finite value
and turns an infinite one into NaN, as 0 times infinity."""
import numpy as np
import pytest

import disco_b200 as db
from test_gpu_caller_capture import make_disk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts", [0, 1])
@pytest.mark.parametrize("prec", [db.PREC_FP64, db.PREC_MIXED])
@pytest.mark.parametrize("base,over", [("c0_kepler2d", {"Num_R": 5}),
                                       ("c1_mhd3d", {"Num_R": 5, "Num_Z": 4, "Constrained_Transport": 1})])
def test_non_finite_cons_of_ghosts(base, over, prec, ts):
    d = make_disk(base, dict(over, Timestep=ts))
    b = db.Batch([d], precision=prec)
    st = b.get_cells()
    ghost = d.real == 0
    rng = np.random.default_rng(3)
    cons = st["cons"].copy()
    cons[ghost] = rng.standard_normal(cons[ghost].shape)
    cons[ghost] = np.where(rng.uniform(size=cons[ghost].shape) < 0.2, np.inf, cons[ghost])
    cons[ghost] = np.where(rng.uniform(size=cons[ghost].shape) < 0.2, -np.inf, cons[ghost])
    st["cons"] = cons
    b.set_cells(**st)
    b.mindt()
    b.timestep()
    got = b.get_cells()["cons"][ghost]
    want = np.where(np.isfinite(cons[ghost]), cons[ghost], np.nan)
    assert np.array_equal(got, want, equal_nan=True)
    assert np.isfinite(b.get_cells()["prim"]).all()
