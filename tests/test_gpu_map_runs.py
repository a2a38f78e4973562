"""Element maps that share a sweep (runs of maps without space charge, and
kick-to-kick sweeps with it) against the same maps launched one by one, which
is what a profiled simulation does.  Both forms apply the same FP32 formulas
to values held in FP32, so they differ by the rounding of fused multiply-adds:
a few 1e-7 an element of each coordinate's spread."""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L
from tests.gpu_runs import COORDS

pytestmark = pytest.mark.gpu


def _run(elems, n, profile, mesh=None, w0=0.75, ranges=((0, -1),)):
    from hpsim_gb300 import HPSim
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.015, num=n, precision="fp32")
    beam.set_waterbag(*L.waterbag_twiss(), 0.0, w0, 201.25, 77)
    beam.set_ref_w(w0)
    beam.set_ref_phi(0.0)
    line = HPSim.BeamLine(elements=elems)
    sc = HPSim.SpaceCharge(*mesh, 0.05, 0) if mesh else None
    sim = HPSim.Simulator(beam, line, sc)
    if profile:
        sim.profile(True)
    launches = HPSim.kernel_launch_count()
    for a, b in ranges:
        sim.simulate(a, b)
    launches = HPSim.kernel_launch_count() - launches
    out = {k: beam._coord(k) for k in COORDS}
    return out, beam._loss(0), beam._loss(1), launches


def _same(a, b, elements):
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])
    live = a[1] == 0
    for k in COORDS:
        spread = a[0][k][live].std() if live.any() else 0.0
        scale = spread + 0.1 * np.abs(a[0][k]).max() / 2 ** 20 + 1e-12
        assert np.abs(a[0][k] - b[0][k]).max() <= 1e-6 * elements * scale, k


def _mixed(n, aperture):
    """drifts, quads of both signs and of none, bunchers, steerers, rotations, dipoles"""
    out = []
    for k in range(n):
        r = k % 11
        if r in (0, 3, 6):
            out.append(L.element(L.DRIFT, f"D{k}", length=0.05, aperture=aperture))
        elif r in (1, 4):
            out.append(L.element(L.QUAD, f"Q{k}", length=0.04, gradient=9.0 if r == 1 else -9.0, aperture=aperture))
        elif r == 7:
            out.append(L.element(L.QUAD, f"Q{k}", length=0.02, gradient=0.0, aperture=aperture))
        elif r == 2:
            out.append(L.element(L.BUNCHER, f"B{k}", voltage=0.01, frequency=201.25, phase=-1.5, aperture=aperture))
        elif r == 5:
            out.append(L.element(L.STEERER, f"S{k}", blh=1e-5, blv=2e-5))
        elif r == 8:
            out.append(L.element(L.ROTATION, f"R{k}", angle=0.1))
        elif r == 9:
            out.append(L.element(L.DIPOLE, f"P{k}", radius=2.0, angle=0.02, edge_in=0.01, edge_out=0.01, half_gap=0.02,
                                 k1=0.4, k2=0.0, field_index=0.5, kinetic_energy=0.75))
        else:
            out.append(L.element(L.QUAD, f"Q{k}", length=0.04, gradient=9.0, aperture=aperture))
    return out


def _channel(n, aperture):
    """the quad channel over and over: a stable lattice of any length"""
    return (L.small_fodo(aperture) * (n // 41 + 1))[:n]


# a drift or quad is two maps: runs of one, two, 16, 17, 256, 257 and more maps
@pytest.mark.parametrize("kind,elements,aperture", [
    (_mixed, 1, 0.0), (_mixed, 2, 0.003), (_mixed, 9, 0.0), (_mixed, 10, 0.003), (_channel, 130, 0.0),
    (_channel, 131, 0.004), (_channel, 300, 0.01)])
@pytest.mark.parametrize("n", [1, 257, 5003])
def test_runs_without_space_charge(kind, elements, aperture, n):
    el = kind(elements, aperture)
    one, many = _run(el, n, True), _run(el, n, False)
    _same(one, many, elements)
    if n == 5003 and elements == 131:
        assert 0 < (many[1] != 0).sum() < n  # some particles are lost on the way
    assert many[3] <= 1 + elements * 2 // 256


@pytest.mark.parametrize("gaps", [1, 16, 40])
def test_runs_with_gaps(gaps):
    el = L.dtl_like(n_gaps=gaps)
    _same(_run(el, 3001, True), _run(el, 3001, False), 2 * gaps)


def test_a_run_ends_with_its_range():
    el = _mixed(20, 0.003)
    whole, parts = _run(el, 1001, False), _run(el, 1001, False, ranges=((0, 4), (5, 5), (6, 19)))
    _same(whole, parts, 20)


@pytest.mark.parametrize("lattice", ["fodo", "dtl", "mixed"])
@pytest.mark.parametrize("n", [4, 255, 1025, 20011])
def test_kick_to_kick_sweeps(lattice, n):
    el = {"fodo": lambda: L.small_fodo()[:6], "dtl": lambda: L.dtl_like(n_gaps=3), "mixed": lambda: _mixed(12, 0.0)}[lattice]()
    one, many = _run(el, n, True, mesh=(32, 128)), _run(el, n, False, mesh=(32, 128))
    assert many[3] < one[3]
    # a kick's rounding: the field table's and the statistics' sums over n particles in FP32, 1e-6 each
    _same(one, many, 10 * len(el))
