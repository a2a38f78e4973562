"""The field network's second input, log(dz gamma / dr), of an FP64 beam is the
FP64 value rounded to BF16, also at energies where 1 - beta^2 cancels in FP32.
The input is read through a network of two layers: the first gives
max(0, input - t), the second passes it on, so the accepted field's interior is
zero exactly where the input is at most t."""
import ctypes as C

import numpy as np
import pytest

from hpsim_gb300 import lattices as L

pytestmark = pytest.mark.gpu
NR, NZ, MASS = 32, 128, 939.294


def _bf16(v):
    import torch
    return float(torch.tensor(v, dtype=torch.float32).bfloat16())


def _bf16_below(v):
    import torch
    b = torch.tensor(v, dtype=torch.float32).bfloat16()
    return float(torch.nextafter(b, torch.tensor(-1e30).bfloat16()))


def _field(gamma, t):
    """(interior of the accepted field, dr, dz, beta) of the first kick"""
    from hpsim_gb300 import HPSim
    from hpsim_gb300._capi import call, dptr
    n, w0 = 4096, MASS * (gamma - 1.0)
    rng = np.random.default_rng(11)
    x, xp, y, yp, phi, w = (rng.standard_normal(n) * s for s in (1e-3, 0.0, 1.3e-3, 0.0, 0.2, 0.0))
    beam = HPSim.Beam(mass=MASS, charge=-1.0, current=0.015, num=n, precision="fp64")
    beam.set_frequency(201.25)
    beam.set_distribution(x, xp, y, yp, phi, w + w0)
    beam.set_ref_w(w0)
    beam.set_ref_phi(0.0)
    sc = HPSim.SpaceCharge(NR, NZ, 0.10, 0)
    w1 = np.zeros((2, 2, 3, 3), np.float32)
    w1[:, 1, 1, 1] = 1.0
    w2 = np.zeros((2, 2, 3, 3), np.float32)
    w2[0, 0, 1, 1] = w2[1, 1, 1, 1] = 1.0
    ws = [(v.view(np.uint32) >> 16).astype(np.uint16) for v in (w1, w2)]  # 0 and 1 are exact in BF16
    bs = [np.full(2, -t, np.float32), np.zeros(2, np.float32)]
    arch, skip = np.array([[2, 2, 1, 1, 1], [2, 2, 1, 1, 0]], np.int32), np.full(2, -1, np.int32)
    ip = C.POINTER(C.c_int)
    call("hps_scheff_set_surrogate", sc.handle, 2, arch.ctypes.data_as(ip), -1, skip.ctypes.data_as(ip),
         (C.c_void_p * 2)(*[v.ctypes.data for v in ws]), (C.c_void_p * 2)(*[v.ctypes.data for v in bs]), NR, NZ, 1.0,
         1e30, 64)
    HPSim.Simulator(beam, HPSim.BeamLine(elements=[L.element(L.DRIFT, "D", length=0.05)]), sc).simulate()
    assert sc.surrogate_stats()[:2] == (1, 0)
    bins, field, mesh = np.empty(NR * NZ), np.empty((NZ + 1) * (NR + 1) * 2), np.empty(7)
    call("hps_scheff_snapshot", sc.handle, 0, dptr(bins), dptr(field), dptr(mesh))
    return field.reshape(NZ + 1, NR + 1, 2)[:NZ, :NR], mesh[2], mesh[3], mesh[4]


@pytest.mark.parametrize("gamma", [1.0008, 2.0, 300.0, 1000.0, 3500.0])
def test_log_aspect_is_rounded_once(gamma):
    _, dr, dz, beta = _field(gamma, 0.0)
    want = _bf16(np.log(dz / np.sqrt(1.0 - beta * beta) / dr))
    assert np.all(_field(gamma, want)[0] == 0.0)  # not above
    assert np.any(_field(gamma, _bf16_below(want))[0] != 0.0)  # not below
