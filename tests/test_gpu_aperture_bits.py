"""Which product an FP32 map rounds when it compares x^2 + y^2 with its
aperture: particles are placed within a few ulp of it, where the choice decides
whether they are lost, and compared with numpy's evaluation.  A short element
and particles without divergence keep x and y as they are."""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L

pytestmark = pytest.mark.gpu
F = np.float32


def _fused(a, b):
    """fma(a, a, round(b b))"""
    return (a.astype(np.float64) ** 2 + (b * b).astype(np.float64)).astype(F)


ELEMENTS = {
    "drift": (lambda ap: L.element(L.DRIFT, "E", length=1e-12, aperture=ap), lambda x, y: _fused(x, y)),
    "quad": (lambda ap: L.element(L.QUAD, "E", length=1e-12, gradient=5.0, aperture=ap), lambda x, y: _fused(y, x)),
    "defocusing quad": (lambda ap: L.element(L.QUAD, "E", length=1e-12, gradient=-5.0, aperture=ap),
                        lambda x, y: _fused(y, x)),
    "quad without gradient": (lambda ap: L.element(L.QUAD, "E", length=1e-12, gradient=0.0, aperture=ap),
                              lambda x, y: _fused(x, y)),
    "buncher": (lambda ap: L.element(L.BUNCHER, "E", voltage=0.0, frequency=201.25, phase=-1.5, aperture=ap),
                lambda x, y: _fused(x, y)),
}


@pytest.mark.parametrize("space_charge", [False, True])
@pytest.mark.parametrize("kind", list(ELEMENTS))
def test_particles_at_the_aperture(kind, space_charge):
    from hpsim_gb300 import HPSim
    n, aperture = 20000, 4.0e-3
    make, radius2 = ELEMENTS[kind]
    a2 = F(aperture * aperture)
    rng = np.random.RandomState(17)
    t = rng.uniform(0.1, 1.4, n)
    x, y = (aperture * np.cos(t)).astype(F), np.zeros(n, F)
    y[:] = np.sqrt(float(a2) - x.astype(np.float64) ** 2).astype(F)
    y = (y.view(np.int32) + rng.randint(-1, 2, n).astype(np.int32)).view(F)
    x[0] = y[0] = 0.0
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.0, num=n, precision="fp32")
    beam.set_frequency(201.25)
    z = np.zeros(n)
    phi = rng.standard_normal(n) * 0.1
    phi[0] = 0.0
    beam.set_distribution(x.astype(np.float64), z, y.astype(np.float64), z, phi, np.full(n, 0.75))
    beam.set_ref_w(0.75)
    beam.set_ref_phi(0.0)
    sc = HPSim.SpaceCharge(32, 128, 0.10, 0) if space_charge else None
    # (a particle's loss is the element's number: 0, the first one's, reads as none)
    HPSim.Simulator(beam, HPSim.BeamLine(elements=[L.element(L.DIAGNOSTICS, "FIRST"), make(aperture)]), sc).simulate()
    assert np.array_equal(beam._coord("x").astype(F), x) and np.array_equal(beam._coord("y").astype(F), y)
    want = radius2(x, y) > a2
    assert np.count_nonzero((radius2(y, x) > a2) != want) > 100  # the choice decides
    assert np.array_equal(beam._loss(0) != 0, want)
