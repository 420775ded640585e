"""Mirror copies on a grid narrower than its ghost zone: with one real annulus
in r, the second ghost layer of a mirrored side copies an annulus of the other
side's first layer.  The layers of both sides then depend on each other, layer
by layer, and every copy equals the reference's sequential walk of it."""
import os

import numpy as np
import pytest

import disco_b200 as db
from test_gpu_zerograd_walk import copy_distant

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
URR, UPP, UZZ = 2, 3, 4


@pytest.mark.parametrize("name,noslip", [("c0_bc_surfaceGravBox", False), ("c0_bc_flowthrough", True)])
def test_one_real_annulus(tmp_path, name, noslip):
    over = {"Num_R": "1", "R_Min": "10.0", "R_Max": "10.2"}
    par = tmp_path / "in.par"
    with open(os.path.join(HERE, "golden", name + ".par")) as f:
        par.write_text("".join("%s %s\n" % (t[0], over[t[0]]) if (t := line.split()) and t[0] in over else line
                               for line in f))
    d = db.Disk.from_files(str(par), os.path.join(db.TEMPLATES, name + ".in"))
    Nr, Nz, Ng = d.Nr, d.Nz, d.Ng
    assert (Nr, Ng[0], Ng[1]) == (5, 2, 2)
    off = np.concatenate([[0], np.cumsum(d.Np)])
    rng = np.random.default_rng(11)
    prim = db.Batch([d]).get_cells()["prim"]
    prim = prim * rng.uniform(0.9, 1.1, prim.shape)
    prim[:, [URR, UZZ]] = rng.uniform(-0.1, 0.1, (len(prim), 2))
    b = db.Batch([d], setup=False)
    for _ in range(20):                    # an order left to chance would show in some of them
        b.restart_cells(prim, d.piph)
        st = b.get_cells()
        for k in range(Ng[2], Nz - Ng[3]):
            cut = [slice(off[j + Nr * k], off[j + Nr * k + 1]) for j in range(Nr)]
            p = [st["prim"][c].copy() for c in cut]

            def copy(j, j1, flip, out_only=False):
                g, s = cut[j], cut[j1]
                x = copy_distant(st["piph"][g], st["dphi"][g], st["piph"][s], st["dphi"][s], p[j1],
                                 d.params.phimax)
                x[:, flip] = -x[:, flip]
                if out_only:
                    x[:, URR] = np.where(x[:, URR] < 0, 0.0, x[:, URR])
                p[j] = x

            flip = [URR, UPP, UZZ] if noslip else [URR]
            for l in range(2):
                copy(1 - l, 2 + l, flip)
                if noslip:                 # the outer side: zero gradient, out of the domain only
                    copy(3 + l, 2 + l, [], True)
                else:
                    copy(3 + l, 2 - l, flip)
            # flowthrough's outer ghosts take a fixed window after the copies
            for j in (0, 1) if noslip else (0, 1, 3, 4):
                assert np.array_equal(st["prim"][cut[j]], p[j]), (j, k)
