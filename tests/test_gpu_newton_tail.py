"""The Newton loop's exit from its tail (grmhd.cuh, c2p_newton): once the
iterate repeats, the remaining iterations are not run.  Prims, iteration
counts and failures equal the C oracle's, which runs them all, for odd and
even tails, tails cut by max_iter and none, at n around a block's cells."""
import numpy as np
import pytest

from oracle import pyc2p
from test_gpu_c2p import _aos, _gr, _soa, _states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 4999])
@pytest.mark.parametrize("nextra,max_iter", [(0, 30), (1, 30), (9, 30), (10, 30), (10, 5), (10, 6), (10, 7),
                                             (10, 12), (10, 13), (31, 100)])
def test_tail_exit_matches_oracle(n, nextra, max_iter):
    for eps in (1e-3, 0.3):
        x, p0, p1 = _states(n, 0.9, eps, seed=5 + nextra)
        orc = pyc2p.C2POracle(metric=1, a=0.9, tol=1e-12, nextra=nextra, max_iter=max_iter)
        gr = _gr(metric="kerr", a=0.9, tol=1e-12, nextra=nextra, max_iter=max_iter)
        cons = orc.prim2cons(p1, x)
        prim_o, it_o, ok_o, _ = orc.cons2prim(cons, x, p0)
        pg = _soa(p0)
        rep = gr.cons2prim(_soa(cons), _soa(x), pg, iters=True)
        np.testing.assert_array_equal(_aos(pg), prim_o)
        np.testing.assert_array_equal(rep["iters"].cpu().numpy().astype(np.int32), it_o)
        assert rep["n_fail"] == int(np.sum(ok_o == 0))
