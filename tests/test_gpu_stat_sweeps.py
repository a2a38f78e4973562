"""The loss-test and moments sweeps of an uncertified space-charge kick
(k32_stat_sweeps) at the edges of its grid: one partly filled cluster, one
full cluster (8 CTAs x 1024 threads x 4 particles), the first particle of a
second cluster, and several clusters.  Tolerances are the FP32 path's stated
ones."""
import numpy as np
import pytest

from tests.test_gpu_fp32 import assert_fp32_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1001, 32768, 32769, 200003])
@pytest.mark.parametrize("late", [True, False])
def test_uncertified_sweeps_match_oracle(oracle, n, late):
    """late: particles beyond <phi> + 3 pi, so the loss test changes the good
    set and the moments are swept again; else particles at the wrap of the
    relative phase only (one sweep)."""
    from hpsim_gb300 import HPSim, lattices as L
    rng = np.random.default_rng(n)
    b0 = oracle.Beam(n)
    b0.set_waterbag(L.waterbag_twiss(), 0.0, 0.75, 201.25, 78)
    x, xp, y, yp, phi, w = (b0.arr(k).copy() for k in ("x", "xp", "y", "yp", "phi", "w"))
    odd = rng.choice(np.arange(1, n), 24, replace=False)
    odd[:2] = (n - 1, n - 2)
    phi[odd[:12]] += 4.0 * np.pi if late else np.pi * 0.9985
    phi[odd[12:]] += np.pi * 0.999
    elems = L.small_fodo()[:3]
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.015, num=n, precision="fp32")
    beam.set_distribution(x, xp, y, yp, phi, w)
    beam.set_ref_w(0.75)
    beam.set_frequency(201.25)
    sc = HPSim.SpaceCharge(32, 128, 0.10, 0)
    sc.set_remesh_threshold(0.0)
    sim = HPSim.Simulator(beam, HPSim.BeamLine(elements=elems), sc)
    sim.enable_monitor(True)
    sim.simulate()
    assert sc.get_counter("stat_sweeps") > 0
    ob = oracle.Beam(n)
    ob.set_distribution(x, xp, y, yp, phi, w)
    ob.set_ref_w(0.75)
    ob.set_frequency(201.25)
    types, params, _ = L.lattice_arrays(elems)
    sp = oracle.Scheff(32, 128, 0.10, 0)
    sp.set(remesh_threshold=0.0)
    mo = oracle.Sim(ob, types, params, sp).simulate().copy()
    assert np.array_equal(beam._loss(0), ob.arr("loss"))
    assert np.array_equal(beam._loss(1), ob.arr("lloss"))
    assert_fp32_close(sim.monitor, mo, "uncertified")
