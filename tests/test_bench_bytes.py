"""bench.py's byte counts of the kernels, each array element once: what k_c2p
reads of the face fluxes under constrained transport."""
import bench


def test_face_fluxes_of_c2p():
    n, nr, nz = 1000, 2003, 1990
    for mixed in (False, True):
        one, two = (bench.kernel_bytes_mhd("k_c2p", first, n, nr, nz, mixed) for first in (True, False))
        # five slots per cell, or the phi faces' slot, one flux per face and wiph
        assert two - one == (nr + nz) * 8 + n * 8 + n * 8 - n * 5 * 8
        for more in (1, 7):
            assert bench.kernel_bytes_mhd("k_c2p", True, n, nr + more, nz, mixed) == one
            assert bench.kernel_bytes_mhd("k_c2p", False, n, nr, nz + more, mixed) == two + more * 8
