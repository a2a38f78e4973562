"""A range's first pass (kernel by kernel), its second (captured) and a replay
give the bits of the same passes with graphs off: both precisions, with
neighbouring bunches, monitors, apertures and a field network attached.  (Pass
by pass: an aperture's loss count stays with the beam and divides the next
pass's sums, as in the reference.  Sizes and meshes of FP32 beams without
these: test_gpu_direct_launch.)"""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L
from tests.gpu_runs import COORDS
from tests.test_gpu_surrogate import _zero_state

pytestmark = pytest.mark.gpu


def _passes(n, precision, lattice, adj, monitor, aperture, network, graph, passes):
    from hpsim_gb300 import HPSim
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.015, num=n, precision=precision)
    beam.set_waterbag(*L.waterbag_twiss(), 0.0, 0.75, 201.25, 5)
    beam.set_ref_w(0.75)
    beam.set_ref_phi(0.0)
    beam.save_initial_beam()
    elems = L.small_fodo(aperture)[:7] if lattice == "fodo" else L.dtl_like(n_gaps=3, aperture=aperture)
    if aperture:
        elems = elems + [L.element(L.APERTURE_C, "APT", aperture=aperture)]
    sc = HPSim.SpaceCharge(32, 128, 0.10, adj)
    sc.set_remesh_threshold(0.0)
    if network:
        sc.set_surrogate(_zero_state(), tol=1e30)  # accepted at every kick
    sim = HPSim.Simulator(beam, HPSim.BeamLine(elements=elems), sc)
    sim.use_graph(graph)
    if monitor:
        sim.enable_monitor(True)
    out = []
    for _ in range(passes):
        beam.restore_initial_beam()
        sim.simulate()
        out.append([beam._coord(k) for k in COORDS] + [beam._loss(0), beam._loss(1)] +
                   ([sim.monitor.copy()] if monitor else []))
    return out


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("lattice,adj,monitor,aperture,network", [
    ("fodo", 0, False, 0.0, False), ("dtl", 1, False, 0.0, False), ("dtl", 0, True, 0.006, False),
    ("fodo", 1, True, 0.006, False), ("fodo", 0, False, 0.0, True), ("dtl", 0, True, 0.0, True)])
@pytest.mark.parametrize("n", [2000, 70001])
def test_every_pass_gives_the_same_bits(precision, lattice, adj, monitor, aperture, network, n):
    got = _passes(n, precision, lattice, adj, monitor, aperture, network, True, 3)
    off = _passes(n, precision, lattice, adj, monitor, aperture, network, False, 3)
    for one, other in zip(got, off):
        for a, b in zip(one, other):
            assert np.array_equal(a, b, equal_nan=True)
