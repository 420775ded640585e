"""Device memory of a 3D constrained-transport batch: what its arrays hold per
cell and per face, with the edge ranks (16 bytes per cell) beside the state and
nothing more per face than the lists, the geometry, the slopes and the fluxes."""
import gc

import pytest
import torch

import disco_b200 as db
from test_gpu_caller_capture import make_disk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [db.PREC_FP64, db.PREC_MIXED])
def test_bytes_of_a_ct_batch(prec):
    d = make_disk("c1_mhd3d", {"Num_R": 160, "Num_Z": 96, "Constrained_Transport": 1})
    N, Np = d.ncell, d.Np.reshape(d.Nz, d.Nr).astype(int)
    F = int((Np[:, 1:] + Np[:, :-1]).sum() + (Np[1:] + Np[:-1]).sum())
    ne = int((Np[1:, 1:] + Np[1:, :-1] + Np[:-1, 1:] + Np[:-1, :-1]).sum())
    r, q = (4, 9) if prec == db.PREC_MIXED else (8, 9)
    cell = (4 * q * r                          # prim and its three slopes
            + 2 * q * 8 + (4 * q if r == 4 else 0)   # cons, RKcons, the carry
            + 4 * 8 + 4 * 4                    # piph, its next value, dphi, wiph; the consume indices
            + 2 * 5 * 8 + 2 * 8 * r + 4 * r    # Phi, RKPhi; edge E and B; the phi faces' four
            + 16)                              # the ranks in the merged edge lines
    face = (2 * 4 + 1 + 3 * 8 + 2 * q * r      # lists, geometry, slope and flux
            + 3 * r + 8 + 1)                   # E, B and E_phi, E dl dt, the flip
    want = N * cell + F * face + ne * 8
    torch.cuda.init()
    gc.collect()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    b = db.Batch([d], precision=prec, setup=False)
    got = free0 - torch.cuda.mem_get_info()[0]
    b.close()
    # 60 allocations rounded up to 2 MiB, the block tables (under 2 bytes per
    # cell or face) and what the library itself loads
    assert got - want < 60 * 2**21 + 2 * (N + F) + 2**26
    assert 48 * N > 60 * 2**21 + 2 * (N + F) + 2**26   # a further 48 bytes per cell would show
