"""FP64 half quads where the focusing angle k length / 4 is below, at and above
the 0.75 that the series serves, with either sign of the gradient and of the
length (a negative length takes particles back), against the oracle.  Both
sides evaluate the same formulas in FP64: the angle to 4 ulp, its functions to
1e-15 relative for angles up to 4, a quad's four steps of two products each;
1e-12 of the largest coordinate leaves room for fifty times that."""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gradient", [18.0, -18.0])
@pytest.mark.parametrize("length", [0.05, 0.2503, 0.6, -0.05, -0.2503, -0.6, -1.2])
def test_half_quads_match_oracle(oracle, length, gradient):
    from hpsim_gb300 import HPSim
    n = 3001
    ob = oracle.Beam(n)
    ob.set_waterbag(L.waterbag_twiss(), 0.0, 0.75, 201.25, 31)
    start = [ob.arr(k).copy() for k in ("x", "xp", "y", "yp", "phi", "w")]
    ob.set_ref_w(0.75)
    ob.set_frequency(201.25)
    elems = [L.element(L.QUAD, "Q", length=length, gradient=gradient)]
    types, params, _ = L.lattice_arrays(elems)
    oracle.Sim(ob, types, params, None).simulate()
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.015, num=n, precision="fp64")
    beam.set_distribution(*start)
    beam.set_ref_w(0.75)
    beam.set_frequency(201.25)
    HPSim.Simulator(beam, HPSim.BeamLine(elements=elems), None).simulate()
    for k in ("x", "xp", "y", "yp", "phi", "w"):
        want = ob.arr(k)
        assert np.abs(beam._coord(k) - want).max() <= 1e-12 * np.abs(want).max(), k
