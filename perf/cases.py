"""Performance cases of the tracking framework: what its users run.

A case is one pass of a user's program: put the initial beam back, track it
through a lattice (or a batch of beams through theirs), and read the results
an analysis or a display needs.  The ranges:

* particles: 1,024 (a knob turned in a control room) to 16,777,216 (a
  production run), odd counts included;
* elements: a short section to the whole 331-element DTL-like linac;
* lattices: the quad channel with a buncher (`small_fodo`), the DTL-like
  linac, the 805 MHz coupled-cavity linac;
* beams of FP64 state (the default precision) and of FP32 state, space charge
  with a solve at every kick or with the default remesh threshold, adjacent
  bunches, apertures, per-element monitors, space charge off;
* one beam, batches of beams of uneven sizes, a set point changed before
  every pass, and the field solve alone on device buffers.

What a program reads after a pass (`read`): "state", the whole particle state
(an FP64 beam's through the coordinate getters as doubles, an FP32 beam's as
phase-space points drawn into device memory, as a display draws them) with
the beam's statistics; "display", the longitudinal phase space and the
statistics; "statistics", sizes, emittances, energies and counts alone, as
a study over many elements or beams reads them.  Over many kicks at low
energy single halo particles follow either of two courses by the last bit of
a mesh size (a particle on the mesh's edge), so long passes there are read by
their statistics.  An FP32 beam's statistics are taken as single-precision
numbers, which is what such a beam holds.
"""
import math

import numpy as np
import torch

from hpsim_gb300 import HPSim, lattices, plotdata
from hpsim_gb300._capi import call, dptr

MASS, CHARGE, CURRENT = 939.294, -1.0, 0.015
# injection energy (MeV), bunch frequency (MHz), SCHEFF mesh and kick interval (m) of each lattice
LATTICES = {
    "fodo": dict(w0=0.75, freq=201.25, mesh=(32, 128), interval=0.10, elements=41),
    "dtl": dict(w0=0.75, freq=201.25, mesh=(32, 128), interval=0.01, elements=331),
    "ccl": dict(w0=100.0, freq=805.0, mesh=(64, 256), interval=0.01, elements=1408),
}
PAIRS = (("x", "xp"), ("y", "yp"), ("phi", "w"))
COORDS = ("x", "xp", "y", "yp", "phi", "w")
# columns of the statistics record: average and rms of each coordinate, emittances
STATISTICS = {"x": (2, 3), "xp": (4, 5), "y": (7, 8), "yp": (9, 10), "phi": (12, 13), "w": (14, 15),
              "emittance_xy": (6, 11), "emittance_z": (16,), "reference": (17, 18)}
COUNTS = (0, 1)


def _case(name, kind="track", lattice="fodo", n=65536, elements=41, precision="fp32", space_charge=True,
          remesh=0.0, adj_bunch=0, aperture=0.0, monitor=False, beams=1, nr=0, nz=0, read="state"):
    c = dict(kind=kind, lattice=lattice, n=n, elements=elements, precision=precision, space_charge=space_charge,
             remesh=remesh, adj_bunch=adj_bunch, aperture=aperture, monitor=monitor, beams=beams,
             nr=nr or LATTICES[lattice]["mesh"][0], nz=nz or LATTICES[lattice]["mesh"][1], read=read)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a control-room model: few particles, a short section, one quad's set point changed before each pass
        _case("knob_1024", kind="knob", n=1024, elements=9),
        # the same through the whole channel with more particles
        _case("knob_20011", kind="knob", n=20011, elements=41, read="statistics"),
        # an online field re-solve on the caller's device buffers, no allocation
        _case("field_32x128", kind="field"),
        # the default beam (FP64) through the quad channel, a solve at every element
        _case("fodo_fp64_65536", n=65536, precision="fp64"),
        # FP64 through the first cells of a linac, limiting apertures, the default remesh threshold, neighbours' fields
        _case("dtl_fp64_150001", lattice="dtl", n=150001, elements=25, precision="fp64", remesh=0.05, adj_bunch=1,
              aperture=0.004),
        # a design study: FP32, an odd count, statistics after every element, the default remesh threshold
        _case("dtl_fp32_100003", lattice="dtl", n=100003, elements=101, remesh=0.05, monitor=True, read="statistics"),
        # the whole linac: what the framework is quoted on
        _case("dtl_fp32_1048576", lattice="dtl", n=1 << 20, elements=331, read="display"),
        # the coupled-cavity linac's larger mesh, several tanks
        _case("ccl_fp32_1000000", lattice="ccl", n=1000000, elements=55),
        # the largest beam: one tank of the coupled-cavity linac
        _case("ccl_fp32_16777216", lattice="ccl", n=1 << 24, elements=11),
        # optics without space charge on a large beam
        _case("optics_fp32_6000001", n=6000001, elements=41, space_charge=False),
        # a set-point scan: beams of uneven sizes (16,384 to 524,288 particles) advanced together
        _case("scan_32", kind="batch", n=92000, beams=32, read="statistics"),
        # equal beams of the coupled-cavity linac with perturbed set points, advanced together
        _case("ccl_batch_6", kind="batch", lattice="ccl", n=262144, elements=22, beams=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("track", "track", "track", "track", "fp64", "fp64", "knob", "batch", "field", "optics"))
    if kind == "field":
        nr, nz = rng.choice(((8, 64), (16, 64), (16, 128), (32, 64), (32, 128), (16, 256)))
        return _case("", kind="field", nr=nr, nz=nz, adj_bunch=rng.choice((0, 0, 1, 2)), n=_log(rng, 1000, 1000000))
    if kind == "knob":
        n, e = _log(rng, 1024, 65536), rng.randrange(5, 42)
        return _case("", kind="knob", n=n, elements=e, read="state" if e <= 7 else "statistics")
    if kind == "optics":
        return _case("", n=_log(rng, 50000, 6000000), elements=rng.randrange(5, 42), space_charge=False)
    if kind == "batch":
        if rng.random() < 0.6:
            return _case("", kind="batch", n=_log(rng, 16384, 131072), beams=rng.randrange(4, 33),
                         elements=rng.randrange(9, 42), read="statistics")
        return _case("", kind="batch", lattice="ccl", n=_log(rng, 16384, 300000), beams=rng.randrange(2, 9),
                     elements=11 * rng.randrange(1, 3))
    remesh, adj = rng.choice((0.0, 0.0, 0.05)), rng.choice((0, 0, 0, 1))
    if kind == "fp64":
        lattice = rng.choice(("fodo", "dtl"))
        n = _log(rng, 2000, 200000)
        e = max(5, min(41, int(4e6 / n)))
        return _case("", lattice=lattice, n=n, elements=e | 1, precision="fp64", remesh=remesh, adj_bunch=adj,
                     aperture=rng.choice((0.0, 0.005)))
    lattice = rng.choice(("fodo", "dtl", "dtl", "ccl", "ccl"))
    n = _log(rng, 4000, 8000000)
    e = int(min({"fodo": 41, "dtl": 200, "ccl": 60}[lattice], max(9, 1.0e8 / n)))
    e = max(11, e // 11 * 11) if lattice == "ccl" else rng.choice((7, e | 1))
    return _case("", lattice=lattice, n=n, elements=e, remesh=remesh, adj_bunch=adj, monitor=rng.random() < 0.25,
                 read="state" if lattice == "ccl" or e <= 7 else "statistics")


def _elements(case):
    """The lattice's first elements; a range ends behind the quad or drift that an RF gap needs after it."""
    e = case["elements"]
    if case["lattice"] == "fodo":
        return lattices.small_fodo(case["aperture"])[:e]
    if case["lattice"] == "dtl":
        return lattices.dtl_like(n_gaps=e // 2, aperture=case["aperture"])
    return lattices.ccl_like(modules=1, tanks=e // 11)


def _waterbag(case, n, seed):
    """A matched 6D waterbag (uniform in a 6-ball), made on the GPU from the seed."""
    spec = LATTICES[case["lattice"]]
    w0, freq = spec["w0"], spec["freq"]
    _, bx, ex, _, by, ey, _, bz, ez = lattices.waterbag_twiss(mass=MASS, w0=w0, freq=freq)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.empty((6, n), dtype=torch.float64, device="cuda")
    for at in range(0, n, 1 << 22):
        m = min(1 << 22, n - at)
        v = torch.randn((6, m), generator=gen, dtype=torch.float64, device="cuda")
        r = torch.rand(m, generator=gen, dtype=torch.float64, device="cuda")
        out[:, at:at + m] = v * (r ** (1.0 / 6.0) / v.square().sum(0).sqrt())
    zmax, zpmax = math.sqrt(ez * bz), math.sqrt(ez / bz)
    wavelength = 100.0 * lattices.CLIGHT / freq  # cm
    out[0] *= 0.01 * math.sqrt(ex * bx)
    out[1] *= math.sqrt(ex / bx)
    out[2] *= 0.01 * math.sqrt(ey * by)
    out[3] *= math.sqrt(ey / by)
    out[4] *= -zmax * 2.0 * math.pi / (lattices.beta_of(w0, MASS) * wavelength)
    out[5] = w0 + 2.0 * w0 * zpmax * out[5]
    out[:5, 0] = 0.0  # particle 0 is the reference particle
    out[5, 0] = w0
    return out.cpu().numpy()


class _Sim:
    """A beam, its lattice, its solver and its simulator, as a program keeps them."""

    def __init__(self, case, n, elems, seed, points=None):
        spec = LATTICES[case["lattice"]]
        self.beam = HPSim.Beam(mass=MASS, charge=CHARGE, current=CURRENT, num=n, precision=case["precision"])
        self.beam.set_frequency(spec["freq"])
        self.beam.set_distribution(*_waterbag(case, n, seed))
        self.beam.set_ref_w(spec["w0"])
        self.beam.set_ref_phi(0.0)
        self.beam.save_initial_beam()
        self.line = HPSim.BeamLine(elements=elems)
        self.solver = None
        if case["space_charge"]:
            self.solver = HPSim.SpaceCharge(case["nr"], case["nz"], spec["interval"], case["adj_bunch"])
            self.solver.set_remesh_threshold(case["remesh"])
        self.sim = HPSim.Simulator(self.beam, self.line, self.solver)
        self.fp64, self.monitor = case["precision"] == "fp64", case["monitor"]
        if self.monitor:
            self.sim.enable_monitor(True)
        self.read = case["read"]
        pairs = {"state": PAIRS, "display": PAIRS[2:], "statistics": ()}[self.read]
        self.points = points  # the display's buffers, by pair
        if points is None:
            self.points = {p: torch.zeros((n, 2), dtype=torch.float32, device="cuda") for p in pairs}

    def draw_points(self):
        for (cx, cy), p in self.points.items():
            plotdata.phase_space(self.beam, cx, cy, device_ptr=p.data_ptr())

    def results(self):
        beam = self.beam
        if self.fp64:
            out = {c: beam._get(c, "all") for c in COORDS}
            out["loss"] = beam.get_losses("t").astype(np.int64)
            out["emittance"] = np.array([beam.get_emittance_x(), beam.get_emittance_y(), beam.get_emittance_z()])
            return out
        self.draw_points()
        out = {a + b: p for (a, b), p in self.points.items()}
        out.update(_statistics(self.sim.monitor if self.monitor else beam.monitor()))
        return out


def _statistics(record):
    """Statistics records as arrays by kind: single-precision numbers and whole counts."""
    record = np.atleast_2d(record)
    out = {k: record[:, list(c)].astype(np.float32) for k, c in STATISTICS.items()}
    out["counts"] = record[:, list(COUNTS)].astype(np.int64)
    return out


def _field_inputs(case, seed):
    """A bunched charge table (a Gaussian in r and z with the noise of n particles) and its mesh."""
    nr, nz = case["nr"], case["nz"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = (torch.arange(nr, device="cuda", dtype=torch.float64) + 0.5) / nr
    z = (torch.arange(nz, device="cuda", dtype=torch.float64) + 0.5) / nz - 0.5
    q = torch.exp(-(z[:, None] / 0.15) ** 2 - (r[None, :] / 0.3) ** 2) * r[None, :]
    mean = q * (case["n"] / q.sum())
    noise = torch.randn((nz, nr), generator=gen, dtype=torch.float64, device="cuda")
    bins = (mean + mean.sqrt() * noise).clamp(min=0.0)
    bins = torch.round(bins * 2.0 ** 20) / 2.0 ** 20  # as the deposit's fixed point holds them
    # dr, dz (m), beta, frequency (MHz), particles, current / mass (A / MeV), adjacent bunches
    mesh = np.array([4.0e-4, 2.0e-4, 0.04, 201.25, case["n"], CURRENT / MASS, case["adj_bunch"]], dtype=np.float64)
    return bins.contiguous(), mesh


def prepare(case, seed):
    HPSim.set_gpu(0)
    kind = case["kind"]
    if kind == "field":
        bins, mesh = _field_inputs(case, seed)
        field = torch.zeros((case["nz"] + 1, case["nr"] + 1, 2), dtype=torch.float64, device="cuda")
        return dict(case=case, bins=bins, mesh=mesh, field=field)
    if kind == "batch":
        sims = []
        rng = np.random.default_rng(seed)
        elems = _elements(case)
        if case["lattice"] == "fodo":
            # sizes spread as the batched scan's: a factor of 32 around the typical size, 16,384 to 524,288
            spread = np.exp(np.linspace(math.log(16384 / 92000), math.log(524288 / 92000), case["beams"]))
            nums = np.clip((case["n"] * spread).astype(np.int64), 4096, 524288)
            scan = [lattices.ScanBeam(int(m), 0, rng.uniform(0.95, 1.05), math.radians(rng.uniform(-3, 3)),
                                      rng.uniform(0.97, 1.03)) for m in nums]
        else:
            scan = lattices.perturbed_beams(case["beams"], case["n"], seed)
        pairs = PAIRS if case["read"] == "state" else ()
        points = {p: torch.zeros((sum(sb.num for sb in scan), 2), dtype=torch.float32, device="cuda") for p in pairs}
        at = 0
        for k, sb in enumerate(scan):
            sims.append(_Sim(case, sb.num, lattices.perturbed(elems, sb), seed * 64 + k,
                             {k: p[at:at + sb.num] for k, p in points.items()}))
            at += sb.num
        return dict(case=case, sims=sims, points=points, batch=HPSim.Batch([s.sim for s in sims]))
    s = _Sim(case, case["n"], _elements(case), seed)
    state = dict(case=case, sims=[s])
    if kind == "knob":
        i = s.line.index("QM00")
        state["knob"] = (i, float(s.line.element(i)[2][lattices.P_GRADIENT]))
        state["turn"] = 0
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "field":
        stream = torch.cuda.current_stream().cuda_stream
        call("hps_scheff_field_noalloc", case["nr"], case["nz"], state["bins"].data_ptr(), dptr(state["mesh"]),
             state["field"].data_ptr(), stream)
        return state["field"]
    sims = state["sims"]
    for s in sims:
        s.beam.restore_initial_beam()
    if case["kind"] == "batch":
        state["batch"].simulate()
        for s in sims:
            s.draw_points()
        out = {a + b: p for (a, b), p in state["points"].items()}
        out.update(_statistics([s.beam.monitor() for s in sims]))
        return out
    s = sims[0]
    if case["kind"] == "knob":
        # the quad's gradient goes up and down by 1 % from pass to pass
        i, g = state["knob"]
        s.line.set_param(i, "gradient", g * (1.01 if state["turn"] % 2 else 1.0))
        state["turn"] += 1
    s.sim.simulate()
    return s.results()


def work(case):
    """Per particle and element the state is read and written once (six
    coordinates, two flags) and about 300 operations are done; per kick the
    field is the sum over all bins at every mesh point, both components."""
    nr, nz = case["nr"], case["nz"]
    solve = 4.0 * (nz + 1) * (nr + 1) * nr * nz
    if case["kind"] == "field":
        return dict(bytes=8.0 * (nr * nz + 2 * (nr + 1) * (nz + 1)), flops=solve)
    if case["kind"] == "batch" and case["lattice"] == "fodo":
        spread = np.exp(np.linspace(math.log(16384 / 92000), math.log(524288 / 92000), case["beams"]))
        total = float(np.clip(case["n"] * spread, 4096, 524288).sum())
    else:
        total = float(case["n"] * case["beams"])
    size = 4 if case["precision"] == "fp32" else 8
    e = case["elements"]
    kicks = case["beams"] * e if case["space_charge"] else 0
    return dict(bytes=total * e * (12 * size + (8 if case["space_charge"] else 4)),
                flops=total * e * (300.0 if case["space_charge"] else 100.0) + kicks * solve)


def _exact_field(case, seed):
    """The sum over all charged rings at every mesh point, from the elliptic-integral fits of the ring's field."""
    bins, mesh = _field_inputs(case, seed)
    nr, nz, adj = case["nr"], case["nz"], case["adj_bunch"]
    dr, dz, beta, freq, num, cur = mesh[:6]
    gm = 1.0 / math.sqrt(1.0 - beta * beta)
    dzg, pl = dz * gm, beta * gm * lattices.CLIGHT / freq
    c1 = 5721.67 * cur / (freq * 1e6 * num)
    f64 = dict(dtype=torch.float64, device="cuda")
    k = torch.arange(nr, **f64)
    rs = (torch.sqrt(0.5 * (k * k + (k + 1) * (k + 1))) * dr)[None, :, None]
    rp = (torch.arange(nr + 1, **f64) * dr)[:, None, None]
    d0 = ((torch.arange(nz, **f64) + 0.5) * dzg)[None, None, :]

    def ring(d):
        b, c = (rp + rs) ** 2, (rp - rs) ** 2
        g = (c + d * d) / (b + d * d)
        h = torch.log(g)
        ee = 1.0 + g * (0.4630106 - 0.2452740 * h + g * (0.1077857 - 0.04125321 * h))
        ek = 1.38629436 - 0.5 * h + g * (0.1119697 - 0.1213486 * h + g * (0.07253230 - 0.02887472 * h))
        a = torch.sqrt(b + d * d)
        er = torch.where(rp != 0, (ek - (rs * rs - rp * rp + d * d) * ee / (c + d * d)) /
                         (2.0 * torch.where(rp != 0, rp, torch.ones_like(rp)) * a), torch.zeros_like(a))
        return er, d * ee / (a * (c + d * d))

    er, ez = ring(d0)
    for i in range(1, adj + 1):
        for s in (-1.0, 1.0):
            e1, e2 = ring(d0 + s * i * pl)
            er, ez = er + e1, ez + e2
    # entries k = -(nz - 1) .. nz of the two-sided table: E_r even, E_z odd about the source's middle
    gr = c1 * torch.cat([er.flip(2), er], 2)
    gz = c1 * torch.cat([-ez.flip(2), ez], 2)
    out = torch.zeros((nz + 1, nr + 1, 2), **f64)
    zs = torch.arange(nz, device="cuda")
    # rows of the sum are cut as the table's partition cuts them on meshes below 1024 bins a part
    total = nr * nz

    def limit(p):
        return (1024 // p) * (total // (1024 // p)) if p <= 1024 else 0

    flat = (zs[:, None] * nr + torch.arange(nr, device="cuda")[None, :])
    body = bins * (flat < limit(nz))
    edge = bins * (flat < limit(nr))
    corner = bins * (flat < (total // 1024) * 1024)
    for zp in range(nz + 1):
        at = zp - zs + nz - 1
        q = body if zp < nz else edge
        out[zp, :, 0] = torch.einsum("psz,zs->p", gr[:, :, at], q)
        out[zp, :, 1] = torch.einsum("psz,zs->p", gz[:, :, at], q)
    at = nz - zs + nz - 1
    out[nz, nr, 0] = (gr[nr][:, at] * corner.T).sum()
    out[nz, nr, 1] = (gz[nr][:, at] * corner.T).sum()
    return out


def _exact_optics(case, seed):
    """Drifts, quads and the buncher in 64 bits on the same particles, no space charge and no apertures."""
    spec = LATTICES[case["lattice"]]
    # the beam takes its state as FP32 values, the energy as offsets from particle 0's
    raw = torch.from_numpy(_waterbag(case, case["n"], seed)).cuda()
    x, xp, y, yp, phi = (raw[i].float().double() for i in range(5))
    w = spec["w0"] + (raw[5] - spec["w0"]).float().double()
    lam = lattices.CLIGHT / spec["freq"]
    q = abs(CHARGE)

    def beta(w):
        g = w / MASS
        return torch.sqrt(g * (g + 2.0)) / (g + 1.0)

    for code, _, p in _elements(case):
        length = float(p[lattices.P_LENGTH])
        if code == lattices.BUNCHER:
            voltage, freq, phase = (float(v) for v in p[3:6])
            lam = lattices.CLIGHT / freq
            g = spec["w0"] / MASS
            btgm = math.sqrt(g * (g + 2.0))
            b = btgm / (g + 1.0)
            con = 2.0 * math.pi * voltage * q / (b * lam * MASS)
            arg = (2.0 * math.pi / (btgm * lam)) ** 2 * (x * x + y * y) * 0.25
            ph = phi * (freq / spec["freq"]) + phase
            dw = q * voltage * torch.cos(ph) * (1.0 + arg * (1.0 + arg * (0.25 + arg / 36.0)))
            bav = beta(w + 0.5 * dw)
            gi, gf = w / MASS, (w + dw) / MASS
            kick = -con * torch.sin(ph) * (1.0 - bav * b) * (0.5 + arg * (0.25 + arg / 24.0)) / bav
            scale = 1.0 / torch.sqrt(gf * (gf + 2.0))
            before = torch.sqrt(gi * (gi + 2.0))
            xp, yp = (xp * before + kick * x) * scale, (yp * before + kick * y) * scale
            w = w + dw
        elif code == lattices.DRIFT:
            x, y = x + length * xp, y + length * yp
            phi = phi + 2.0 * math.pi * length / (lam * beta(w))
        else:
            qg = float(p[lattices.P_GRADIENT]) * CHARGE
            for _ in range(2):
                g = w / MASS
                bg = torch.sqrt(g * (g + 2.0) * (1.0 + xp * xp + yp * yp))
                k = torch.sqrt(abs(qg) / (bg * MASS) * lattices.CLIGHT)
                kd = 0.25 * length * k
                c, s, ch, sh = torch.cos(kd), torch.sin(kd), torch.cosh(kd), torch.sinh(kd)
                for _ in range(2):
                    fx = (c * x + s / k * xp, -s * k * x + c * xp) if qg > 0 else (ch * x + sh / k * xp, sh * k * x + ch * xp)
                    fy = (ch * y + sh / k * yp, sh * k * y + ch * yp) if qg > 0 else (c * y + s / k * yp, -s * k * y + c * yp)
                    (x, xp), (y, yp) = fx, fy
                phi = phi + math.pi * length / (lam * beta(w))
    g0 = w[0] / MASS
    bg0 = torch.sqrt(g0 * (g0 + 2.0))
    turn = 2.0 * math.pi
    rel = torch.remainder(phi - phi[0] + math.pi, turn) - math.pi

    def moments(a):
        return [a.mean(), a.std(correction=0)]

    def emittance(a, b):
        a, b = a - a.mean(), b - b.mean()
        return torch.sqrt((a * a).mean() * (b * b).mean() - (a * b).mean() ** 2)

    out = {"xxp": torch.stack([x, xp], 1), "yyp": torch.stack([y, yp], 1), "phiw": torch.stack([phi, w], 1)}
    record = {"x": moments(x), "xp": moments(xp), "y": moments(y), "yp": moments(yp), "phi": moments(rel),
              "w": moments(w), "emittance_xy": [bg0 * emittance(x, xp), bg0 * emittance(y, yp)],
              "emittance_z": [emittance(rel, w)], "reference": [w[0], phi[0]]}
    out.update({k: torch.stack(v)[None] for k, v in record.items()})
    out["counts"] = None
    return out


def exact(case, seed):
    if case["kind"] == "field":
        return _exact_field(case, seed)
    if case["kind"] == "track" and not case["space_charge"]:
        return _exact_optics(case, seed)
    return None  # space charge on a beam: every element solves the field of all particles, too long in plain torch
