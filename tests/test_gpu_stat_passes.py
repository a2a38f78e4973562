"""Beam statistics records at the sizes where the reduction passes change
shape (one particle, partial warps and blocks, the block-count tiers), against
plain FP64 numpy sums."""
import math

import numpy as np
import pytest

from hpsim_gb300 import HPSim

pytestmark = pytest.mark.gpu

MASS, W0 = 939.294, 0.75
SCALE = np.array([2e-3, 3e-3, 1e-3, 2e-3, 0.4, 5e-3])


def _record(c):
    """averages, sigmas and emittances of the record's layout (x, y, relative phase)"""
    rel = np.remainder(c[4] - c[4, 0] + math.pi, 2 * math.pi) - math.pi
    g0 = c[5, 0] / MASS
    bg = math.sqrt(g0 * (g0 + 2.0))
    out, tol = [], []
    for a, b, f in ((c[0], c[1], bg), (c[2], c[3], bg), (rel, c[5], 1.0)):
        sa, sb = a.std(), b.std()
        cov = ((a - a.mean()) * (b - b.mean())).mean()
        out += [a.mean(), sa, b.mean(), sb, f * math.sqrt(max(sa * sa * sb * sb - cov * cov, 0.0))]
        tol += [sa, sa, sb, sb, f * sa * sb]
    return np.array(out), np.array(tol)


# FP64 W is summed with its offset of W0: sigma_W^2 as a difference loses
# (W0 / sigma_W)^2 = 2e4 of the 1e-16 a term, 1e-11 with the sums' own rounding.
# FP32: a thread's and a warp's sums of up to a few dozen terms, 2^-24 each
@pytest.mark.parametrize("precision,rel", [("fp64", 1e-10), ("fp32", 2e-5)])
@pytest.mark.parametrize("n", [33, 255, 257, 1025, 304 * 256, 304 * 256 + 1, 311299])
def test_statistics_record_matches_numpy(n, precision, rel):
    rng = np.random.default_rng(n)
    c = rng.standard_normal((6, n)) * SCALE[:, None]
    c[5] += W0
    c[:5, 0] = 0.0
    c[5, 0] = W0
    if precision == "fp32":  # the values the beam holds
        c[:5] = c[:5].astype(np.float32)
        c[5] = W0 + (c[5] - W0).astype(np.float32)
    beam = HPSim.Beam(mass=MASS, charge=-1.0, current=0.015, num=n, precision=precision)
    beam.set_distribution(*c)
    beam.set_ref_w(W0)
    beam.set_ref_phi(0.0)
    want, scale = _record(c)
    rec = beam.monitor()
    assert rec[0] == n and rec[1] == n
    assert np.all(np.abs(rec[2:17] - want) <= rel * scale), (rec[2:17] - want) / scale
    assert rec[17] == pytest.approx(W0, rel=1e-7)
    ex, ez = beam.get_emittance_x(), beam.get_emittance_z()
    assert abs(ex - want[4]) <= rel * scale[4] and abs(ez - want[14]) <= rel * scale[14]
