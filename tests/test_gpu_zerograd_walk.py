"""The zero-gradient ghost copy (k_zerograd: every thread walks its own ghost
cells from a guessed start, wrong guesses walked again in order; the layers of
a side chained in one block) against set_cells_copy_distant restated here as
the reference's sequential walk, bit for bit, from the source annulus's own
downloaded prims: annuli of fewer and more cells than a block, unequal
neighbours, edges that coincide, an annulus whose first cell lies anywhere."""
import os

import numpy as np
import pytest

import disco_b200 as db
from disco_b200.workloads import write_par

pytestmark = pytest.mark.gpu


def copy_distant(gp, gd, sp, sd, prim, pmax):
    """boundary_functions.c:90-158 for one ghost annulus (edges gp, widths gd)."""
    n1 = len(sp)

    def signed(x):
        while x < -.5 * pmax:
            x += pmax
        while x > .5 * pmax:
            x -= pmax
        return x
    i1 = 0
    phi0 = gp[0] - gd[0]
    for k in range(n1):
        dp = signed(sp[k] - phi0)
        if dp > 0 and dp - sd[k] <= 0.0:
            i1 = k
            break
    out = np.zeros((len(gp), prim.shape[1]))
    for i in range(len(gp)):
        hi, lo = gp[i], gp[i] - gd[i]
        acc = np.zeros(prim.shape[1])
        while True:
            h1, l1 = sp[i1], sp[i1] - sd[i1]
            while h1 < lo:
                h1 += pmax
                l1 += pmax
            while l1 > hi:
                h1 -= pmax
                l1 -= pmax
            acc = acc + prim[i1] * ((hi if hi < h1 else h1) - (lo if lo > l1 else l1))
            i1 = (i1 + 1) % n1
            if not h1 < hi:
                break
        i1 = (i1 - 1) % n1
        out[i] = acc / gd[i]
    return out


def _edges(n, how, pmax, rng):
    if how == "ties":                     # every annulus's edges on the same grid of angles
        e = np.arange(n) * (pmax / n)
    elif how == "ragged":                 # widths from 0.2 to 1.8 of the mean
        w = rng.uniform(0.2, 1.8, n)
        e = (np.cumsum(w) / w.sum() + rng.uniform()) * pmax
    else:
        e = (np.arange(n) + rng.uniform()) * (pmax / n)
    e = np.where(e > pmax, e - pmax, e)
    e = np.where(e < 0, e + pmax, e)
    return np.roll(e, rng.integers(n))


@pytest.mark.parametrize("how", ["ties", "ragged", "even"])
@pytest.mark.parametrize("base,nr,nz,aspect", [("c0_kepler2d", 6, 1, 1.0), ("c1_mhd3d", 7, 4, 1.34),
                                               ("c1_mhd3d", 9, 3, 0.11)])
def test_zerograd_equals_sequential_walk(base, nr, nz, aspect, how):
    over = {"Num_R": nr, "aspect": aspect}
    if nz > 1:
        over["Num_Z"] = nz
    p = write_par(over, base=base)
    disk = db.Disk.from_files(p, os.path.join(db.TEMPLATES, "c0_zerograd.in" if nz == 1 else "c1_mhd3d.in"))
    os.unlink(p)
    assert nr < 9 or disk.Np.max() > 256
    rng = np.random.default_rng(nr)
    pmax = disk.params.phimax
    off = np.concatenate([[0], np.cumsum(disk.Np)])
    piph = np.concatenate([_edges(int(n), how, pmax, rng) for n in disk.Np])
    prim = db.Batch([disk]).get_cells()["prim"]
    prim = prim * rng.uniform(0.9, 1.1, prim.shape)
    b = db.Batch([disk], setup=False)
    b.restart_cells(prim, piph)
    st = b.get_cells()
    Nr, Nz, Ng = disk.Nr, disk.Nz, disk.Ng
    cells = lambda j, k: slice(off[j + Nr * k], off[j + Nr * k + 1])
    pairs = []
    for k in range(Nz):
        pairs += [(j, k, j + 1, k) for j in range(Ng[0])]
        pairs += [(j, k, j - 1, k) for j in range(Nr - Ng[1], Nr)]
    if Nz > 1:
        # the corners are copied again by the z pass
        z = [(j, k, j, k + 1) for j in range(Nr) for k in range(Ng[2])]
        z += [(j, k, j, k - 1) for j in range(Nr) for k in range(Nz - Ng[3], Nz)]
        done = {q[:2] for q in z}
        pairs = [q for q in pairs if q[:2] not in done] + z
    assert pairs
    for j, k, j1, k1 in pairs:
        g, s = cells(j, k), cells(j1, k1)
        want = copy_distant(st["piph"][g], st["dphi"][g], st["piph"][s], st["dphi"][s], st["prim"][s], pmax)
        assert np.array_equal(st["prim"][g], want), (j, k)
