"""The FP64 field solve on meshes at the edges of its kernels' rules (lane
groups below 32 source radii, several lanes' passes above, the smallest and
the largest table an SM holds, the meshes just outside) against the oracle's
table stage: 1e-12 of the largest component, the rounding of sums of up to
8,192 terms of either sign."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_scheff_field import field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nz", [(16, 64), (32, 32), (8, 128), (4, 256), (2, 512), (64, 16), (128, 8), (256, 4),
                                   (16, 128), (32, 128), (64, 128), (256, 32), (32, 256), (16, 512),
                                   (16, 32), (8, 64), (32, 512), (64, 256)])
@pytest.mark.parametrize("adj", [0, 1])
def test_field_against_oracle(oracle, nr, nz, adj):
    rng = np.random.default_rng(nr * 1000 + nz)
    bins = rng.uniform(0.0, 5.0, nr * nz) * (rng.uniform(size=nr * nz) > 0.3)
    bins = np.round(bins * 2.0 ** 20) / 2.0 ** 20  # exact in the solver's 2^-36 fixed point
    mesh = np.array([4.0e-4, 2.0e-4, 0.05, 201.25, 65536, 1.6e-5, float(adj)])
    f = field(nr, nz, bins, mesh)
    s = oracle.Scheff(nr, nz, 0.01, 0)
    s.s.dr, s.s.dz = mesh[0], mesh[1]
    oracle.lib().orc_scheff_green_table(s.h, mesh[2], mesh[3], int(mesh[4]), mesh[5], int(mesh[6]))
    C.memmove(s.s.bin, bins.ctypes.data, bins.nbytes)
    oracle.lib().orc_scheff_contract(s.h)
    _, _, ref = s.tables()
    for c in (0, 1):
        a, b = f[c::2], ref[c::2]
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), (c, np.abs(a - b).max() / np.abs(b).max())


def test_single_charges_reach_every_point(oracle):
    """One charged bin at a time: every point sees it at its own distance."""
    nr, nz = 32, 64
    mesh = np.array([4.0e-4, 2.0e-4, 0.05, 201.25, 65536, 1.6e-5, 0.0])
    for zs, rs in ((0, 0), (0, 31), (15, 7), (16, 8), (31, 31), (32, 0), (47, 16), (48, 17), (63, 0), (63, 31)):
        bins = np.zeros(nr * nz)
        bins[zs * nr + rs] = 3.0
        s = oracle.Scheff(nr, nz, 0.01, 0)  # its sum adds to the table it holds
        s.s.dr, s.s.dz = mesh[0], mesh[1]
        oracle.lib().orc_scheff_green_table(s.h, mesh[2], mesh[3], int(mesh[4]), mesh[5], 0)
        C.memmove(s.s.bin, bins.ctypes.data, bins.nbytes)
        oracle.lib().orc_scheff_contract(s.h)
        _, _, ref = s.tables()
        f = field(nr, nz, bins, mesh)
        assert np.abs(f - ref).max() <= 1e-12 * np.abs(ref).max(), (zs, rs)
