"""FP32 particles so near the axis that x^2 + y^2 is subnormal (|x| between
about 1e-23 and 1e-19 m): they pass an RF gap and a kick as the ones on the
axis do.  Away from the axis's own scale nothing depends on such an offset, so
the survivors' coordinates agree with an on-axis particle's to FP32 rounding of
the spread (1e-6)."""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L
from tests.gpu_runs import COORDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("space_charge", [False, True])
@pytest.mark.parametrize("lattice", ["dtl", "ccl"])
@pytest.mark.parametrize("offset", [1e-22, 1e-20, 3e-20, 0.9e-19])
def test_subnormal_radius(lattice, offset, space_charge):
    from hpsim_gb300 import HPSim
    n, w0, freq = 1024, (0.75 if lattice == "dtl" else 100.0), (201.25 if lattice == "dtl" else 805.0)
    elems = L.dtl_like(n_gaps=1) if lattice == "dtl" else L.ccl_like(modules=1, tanks=1)
    rng = np.random.default_rng(3)
    x, xp, y, yp, phi, w = (rng.standard_normal(n) * s for s in (1e-3, 1e-3, 1e-3, 1e-3, 0.1, 1e-3))
    w += w0
    for c, v in zip((x, xp, y, yp, phi, w), (0.0, 0.0, 0.0, 0.0, 0.0, w0)):
        c[0] = v
        c[100:104] = v
    x[100], y[101], x[102], y[102] = offset, -offset, offset, offset  # 103 stays on the axis
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.015, num=n, precision="fp32")
    beam.set_frequency(freq)
    beam.set_distribution(x, xp, y, yp, phi, w)
    beam.set_ref_w(w0)
    beam.set_ref_phi(0.0)
    sc = HPSim.SpaceCharge(32, 128, 0.05, 0) if space_charge else None
    HPSim.Simulator(beam, HPSim.BeamLine(elements=elems), sc).simulate()
    assert not beam._loss(0).any()
    for k in COORDS:
        c = beam._coord(k)
        spread = c.std()
        assert np.isfinite(c).all()
        assert np.abs(c[100:103] - c[103]).max() <= 1e-6 * spread, k
