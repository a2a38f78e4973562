"""The wide form of the FP32 ring convolution (meshes of 32 k source radii,
32 to 256 rows) at the edges of its blocks (33 field rows, 11 points a warp,
quarters of the source rows) and on either side of its dispatch line, against
the FP64 table stage: the FP32 path's 2e-5 of the largest component."""
import numpy as np
import pytest

from tests.test_gpu_scheff_field import _bunched, _close_per_component, field, field_f32_kernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nz", [(32, 32), (32, 64), (64, 32), (64, 64), (64, 128), (256, 32), (128, 256),
                                   (16, 64), (32, 512), (32, 16)])
@pytest.mark.parametrize("adj", [0, 1])
def test_field_against_fp64(nr, nz, adj):
    mesh = np.array([4.0e-4, 2.0e-4, 0.05, 201.25, 65536, 1.6e-5, float(adj)])
    rng = np.random.default_rng(nr * 1000 + nz)
    for bins in (_bunched(nr, nz), rng.uniform(0.0, 5.0, nr * nz) * (rng.uniform(size=nr * nz) > 0.3)):
        _close_per_component(field_f32_kernel(nr, nz, bins, mesh, 1), field(nr, nz, bins, mesh), 2e-5)


def test_single_charges_reach_every_point():
    """One charged bin at a time, at the corners and the middle of the mesh:
    every point of the table against the FP64 stage."""
    nr, nz = 32, 64
    mesh = np.array([4.0e-4, 2.0e-4, 0.05, 201.25, 65536, 1.6e-5, 0.0])
    for zs, rs in ((0, 0), (0, 31), (63, 0), (63, 31), (15, 7), (16, 8), (31, 16), (32, 17)):
        bins = np.zeros(nr * nz)
        bins[zs * nr + rs] = 3.0
        _close_per_component(field_f32_kernel(nr, nz, bins, mesh, 1), field(nr, nz, bins, mesh), 2e-5)


def test_solvers_choice():
    """Left to choose, a solver takes CUDA cores up to nr nz = 8192; told, it
    takes what it is told."""
    from hpsim_gb300 import HPSim
    for nr, nz, tc in ((32, 128, 0), (64, 128, 0), (64, 256, 1), (16, 256, 1), (8, 64, 0)):
        sc = HPSim.SpaceCharge(nr, nz, 0.1, 0)
        assert sc.get_counter("tensor_cores") == tc
    sc = HPSim.SpaceCharge(32, 128, 0.1, 0)
    sc.set_contraction("tensor")
    assert sc.get_counter("tensor_cores") == 1
    sc.set_contraction("cuda")
    assert sc.get_counter("tensor_cores") == 0
