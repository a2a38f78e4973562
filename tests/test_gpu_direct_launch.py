"""A range's first pass is launched kernel by kernel, its second as a captured
graph: the same kernels, so the same bits, on either side of the sizes where
the direct form changes (one deposit block an SM, the particles up to which
kernels are scheduled ahead); and a range that ends in a lattice error leaves
the beam as it was."""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L
from tests.gpu_runs import COORDS

pytestmark = pytest.mark.gpu


def _sim(n, elems, mesh=(32, 128), precision="fp32"):
    from hpsim_gb300 import HPSim
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.015, num=n, precision=precision)
    beam.set_waterbag(*L.waterbag_twiss(), 0.0, 0.75, 201.25, 5)
    beam.set_ref_w(0.75)
    beam.set_ref_phi(0.0)
    beam.save_initial_beam()
    line = HPSim.BeamLine(elements=elems)
    sc = HPSim.SpaceCharge(*mesh, 0.10, 0)
    sc.set_remesh_threshold(0.0)
    return beam, line, sc, HPSim.Simulator(beam, line, sc)


@pytest.mark.parametrize("mesh", [(32, 128), (64, 256)])
@pytest.mark.parametrize("n", [5, 1024, 1025, 38912, 38913, 65536, 65537])
def test_direct_pass_equals_graph_pass(n, mesh):
    elems = L.dtl_like(n_gaps=2) if mesh == (64, 256) else L.small_fodo()[:5]
    beam, line, sc, sim = _sim(n, elems, mesh)
    got = []
    for _ in range(4):  # direct, captured, replayed, replayed
        beam.restore_initial_beam()
        sim.simulate()
        got.append([beam._coord(k) for k in COORDS] + [beam._loss(0), beam._loss(1)])
    for later in got[1:]:
        for a, b in zip(got[0], later):
            assert np.array_equal(a, b, equal_nan=True)


def test_set_points_that_change_between_passes():
    """Every pass has new inputs: each equals a fresh simulator's pass."""
    elems = L.small_fodo()[:5]
    beam, line, sc, sim = _sim(2000, elems)
    i = line.index("QM00")
    for g in (18.0, 18.2, 18.0, 17.9, 17.9, 18.2):
        beam.restore_initial_beam()
        line.set_param(i, "gradient", g)
        sim.simulate()
        ref, rline, rsc, rsim = _sim(2000, elems)
        rline.set_param(i, "gradient", g)
        ref.restore_initial_beam()
        rsim.simulate()
        for k in COORDS:
            assert np.array_equal(beam._coord(k), ref._coord(k)), (g, k)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_a_lattice_error_leaves_the_beam_alone(precision):
    elems = L.dtl_like(n_gaps=2)
    broken = elems[:3] + [elems[1]]  # quad, gap, quad, gap: no quad behind the last gap
    beam, line, sc, sim = _sim(1000, broken, precision=precision)
    before = [beam._coord(k) for k in COORDS]
    with pytest.raises(Exception, match="quad|gap"):
        sim.simulate()
    for a, k in zip(before, COORDS):
        assert np.array_equal(a, beam._coord(k)), k
