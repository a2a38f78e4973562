"""A run of FP32 maps that takes several launches (256 maps each, 64 where an RF
gap's second half is among them) gives the particles what one launch a map does,
whatever map a launch begins with: drifts and quads share 1/beta of the particles
while nothing changes the energies, and a launch has to form it for itself."""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L
from tests.test_gpu_map_bits import _equal, _state

pytestmark = pytest.mark.gpu


def _drift(k):
    return L.element(L.DRIFT, f"D{k}", length=0.002)


def _odd(kind):
    if kind == "steerer":
        return L.element(L.STEERER, "ODD", blh=1e-5, blv=2e-5)
    if kind == "rotation":
        return L.element(L.ROTATION, "ODD", angle=0.1)
    return L.element(L.DIPOLE, "ODD", radius=2.0, angle=0.02, edge_in=0.01, edge_out=0.01, half_gap=0.02, k1=0.4,
                     k2=0.0, field_index=0.5, kinetic_energy=0.75)


def _line(kind, at, gap):
    """Maps 0 .. at - 1 (drifts are two maps, a steerer one), then the odd map,
    the odd dipole's second half where kind says so, then drifts and quads."""
    out = L.dtl_like(n_gaps=1) if gap else []  # six maps
    fill = at - (6 if gap else 0) - (1 if kind == "dipole second half" else 0)
    if fill % 2:
        out.append(L.element(L.STEERER, "PAD", blh=1e-5, blv=2e-5))
        fill -= 1
    out += [_drift(k) for k in range(fill // 2)] + [_odd(kind)]
    for k in range(3):
        out += [_drift(1000 + k), L.element(L.QUAD, f"QX{k}", length=0.04, gradient=9.0)]
    return out


@pytest.mark.parametrize("kind", ["steerer", "rotation", "dipole first half", "dipole second half"])
@pytest.mark.parametrize("at,gap", [(256, False), (255, False), (512, False), (64, True), (128, True), (63, True)])
def test_split_behind_any_map(kind, at, gap):
    from hpsim_gb300 import HPSim
    got = []
    for profile in (True, False):  # a profiled simulation launches every map by itself
        beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.015, num=2001, precision="fp32")
        beam.set_waterbag(*L.waterbag_twiss(), 0.0, 0.75, 201.25, 7)
        beam.set_ref_w(0.75)
        beam.set_ref_phi(0.0)
        sim = HPSim.Simulator(beam, HPSim.BeamLine(elements=_line(kind, at, gap)), None)
        sim.profile(profile)
        sim.simulate()
        got.append(_state(beam))
    assert np.ptp(got[0]["w"]) > 1e-3  # the energies differ, so 1/beta does
    _equal(*got)
