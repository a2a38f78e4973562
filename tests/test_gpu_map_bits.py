"""An FP32 map or kick gives a particle the same bits in every launch that it
shares: alone, as one map a launch (which a profiled simulation runs), in a run
of maps, in the sweep from kick to kick, and as a beam of a batch.  Beyond a
space-charge kick the particles' last bits decide which of its two fields a
particle at the mesh's edge gets, so equality is exact."""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L
from tests.gpu_runs import COORDS
from tests.test_gpu_map_runs import _mixed

pytestmark = pytest.mark.gpu
LATTICES = {
    "fodo": (lambda ap: L.small_fodo(ap)[:21], 0.75, 201.25, (32, 128)),
    "dtl": (lambda ap: L.dtl_like(n_gaps=12, aperture=ap), 0.75, 201.25, (32, 128)),
    "ccl": (lambda ap: L.ccl_like(modules=1, tanks=2), 100.0, 805.0, (64, 256)),
    "mixed": (lambda ap: _mixed(22, ap), 0.75, 201.25, (32, 128)),
}


def _sim(lattice, n, seed, aperture, mesh, adj=0):
    from hpsim_gb300 import HPSim
    elems, w0, freq, nrnz = LATTICES[lattice]
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.015, num=n, precision="fp32")
    beam.set_frequency(freq)
    beam.set_waterbag(*L.waterbag_twiss(mass=939.294, w0=w0, freq=freq), 0.0, w0, freq, seed)
    beam.set_ref_w(w0)
    beam.set_ref_phi(0.0)
    sc = HPSim.SpaceCharge(*nrnz, 0.05, adj) if mesh else None
    if mesh:
        sc.set_remesh_threshold(0.0)
    sim = HPSim.Simulator(beam, HPSim.BeamLine(elements=elems(aperture)), sc)
    return sim, beam


def _state(beam):
    out = {k: beam._coord(k) for k in COORDS}
    out["loss"], out["lloss"] = beam._loss(0), beam._loss(1)
    return out


def _equal(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), (k, np.flatnonzero(a[k] != b[k])[:5])


@pytest.mark.parametrize("lattice", list(LATTICES))
@pytest.mark.parametrize("mesh,adj", [(False, 0), (True, 0), (True, 1)])
@pytest.mark.parametrize("n,aperture", [(1000, 0.0), (20011, 0.006)])
def test_one_by_one_and_together(lattice, mesh, adj, n, aperture):
    got = []
    for profile in (True, False):
        sim, beam = _sim(lattice, n, 5, aperture, mesh, adj)
        sim.profile(profile)
        sim.simulate()
        got.append(_state(beam))
    _equal(*got)


@pytest.mark.parametrize("lattice", list(LATTICES))
@pytest.mark.parametrize("lockstep", [False, True])
def test_alone_and_in_a_batch(lattice, lockstep):
    from hpsim_gb300 import HPSim
    sizes = (1000, 5003)
    alone = []
    for k, n in enumerate(sizes):
        sim, beam = _sim(lattice, n, 20 + k, 0.006, False)
        sim.simulate()
        alone.append(_state(beam))
    pairs = [_sim(lattice, n, 20 + k, 0.006, False) for k, n in enumerate(sizes)]
    batch = HPSim.Batch([s for s, _ in pairs])
    batch.set_lockstep(lockstep)
    batch.simulate()
    assert batch.last_mode()[0] == ("lockstep" if lockstep else "graphs")
    for want, (_, beam) in zip(alone, pairs):
        _equal(want, _state(beam))
