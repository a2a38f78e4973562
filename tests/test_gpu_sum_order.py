"""The order of the sums behind a kick's mesh, to the bit.

The mesh's radius is three rms heights of the beam; a particle at its edge is
kicked from either side by the edge's last bit, so the FP32 sums of y and y^2
have one order whatever kernel takes them: blocks of 256 threads (a particle
in every blocks x 256 each), shuffle trees, warps in order, then the blocks in
32 chains and a tree.  Here that order is taken by numpy in FP32 and compared
with the solver's mesh, at the edges of the blocks (1,024 particles fill one,
311,296 all of two an SM, 155,648 all of one).  The beam stands still (no
divergence, one energy, no current), so that every kick sees the particles as
they were set: the first kick's sums come from a half element's sweep, the
later ones' from the sweep around a kick.  Both sides round the same
operations, so they agree exactly."""
import numpy as np
import pytest

from hpsim_gb300 import lattices as L

pytestmark = pytest.mark.gpu
F = np.float32


def _tree(v):
    """lane 0 of a shuffle tree over the last axis (32 lanes)"""
    for off in (16, 8, 4, 2, 1):
        v = v[..., :off] + v[..., off:2 * off]
    return v[..., 0]


def _fma(a, b, c):
    return F(np.float64(a) * np.float64(b) + np.float64(c))


def _block_warps(v, blocks, square):
    """Warp sums of `blocks` blocks: every thread adds its particles in turn.
    square: None the values, "mul" their squares rounded first, "fma" fused."""
    rounds = -(-len(v) // (256 * blocks))
    v = np.concatenate([v, np.zeros(rounds * blocks * 256 - len(v), F)]).reshape(rounds, blocks, 256)
    acc = np.zeros((blocks, 256), F)
    for r in v:
        if square is None:
            acc = acc + r
        elif square == "mul":
            acc = acc + r * r
        else:
            acc = (r.astype(np.float64) ** 2 + acc.astype(np.float64)).astype(F)
    return _tree(acc.reshape(blocks, 8, 32))


def _grid_sum(v, blocks, square=None):
    warps = _block_warps(v, blocks, square)
    part = np.zeros(blocks, F)
    for w in range(8):
        part = part + warps[:, w]
    chains = np.zeros(32, F)
    for b in range(0, blocks, 32):
        row = part[b:b + 32]
        chains[:len(row)] = chains[:len(row)] + row
    return _tree(chains)


def _single_block_sum(v, square=None):
    """the second sweep: one block, its warps in FP64"""
    s = 0.0
    for w in _block_warps(v, 1, square)[0]:
        s += float(w)
    return F(s)


def _edge(sy, syy, n):
    isv = F(1.0) / F(n)
    ya = F(sy * isv)
    return F(3.0) * np.sqrt(_fma(-ya, ya, F(syy * isv)))


def _blocks(n, per_sm):
    return min(max(-(-n // 1024), 1), per_sm * 152)


def _beam(n, y, phi):
    from hpsim_gb300 import HPSim
    beam = HPSim.Beam(mass=939.294, charge=-1.0, current=0.0, num=n, precision="fp32")
    z = np.zeros(n)
    x = np.random.default_rng(n).standard_normal(n) * 1e-3
    x[0] = 0.0
    beam.set_distribution(x, z, y.astype(np.float64), z, phi, np.full(n, 0.75))
    beam.set_ref_w(0.75)
    beam.set_ref_phi(0.0)
    beam.set_frequency(201.25)
    sc = HPSim.SpaceCharge(32, 128, 0.10, 0)
    sc.set_remesh_threshold(0.0)
    return beam, sc


def _inputs(n, seed):
    rng = np.random.default_rng(1000 * seed + n)
    y = (rng.standard_normal(n) * 1.7e-3 + 3e-4).astype(F)
    y[0] = 0.0
    phi = rng.standard_normal(n) * 0.2
    phi[0] = 0.0
    return y, phi


def _line(drifts):
    return [L.element(L.DRIFT, f"D{k}", length=0.05) for k in range(drifts)]


def _mesh_edge(sc):
    from hpsim_gb300._capi import call, dptr
    bins, field, mesh = np.empty(32 * 128), np.empty(129 * 33 * 2), np.empty(7)
    call("hps_scheff_snapshot", sc.handle, 1, dptr(bins), dptr(field), dptr(mesh))
    return F(mesh[2]) * F(32)


SIZES = [1000, 1025, 5001, 40000, 155649, 311296, 311297, 700001]


@pytest.mark.parametrize("drifts", [1, 3])
@pytest.mark.parametrize("n", SIZES)
def test_certified_sums(n, drifts):
    from hpsim_gb300 import HPSim
    for seed in range(3):
        y, phi = _inputs(n, seed)
        beam, sc = _beam(n, y, phi)
        HPSim.Simulator(beam, HPSim.BeamLine(elements=_line(drifts)), sc).simulate()
        assert sc.get_counter("stat_sweeps") == 0
        g = _blocks(n, 2)
        assert _mesh_edge(sc) == _edge(_grid_sum(y, g), _grid_sum(y, g, "mul"), n)


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("n", SIZES)
def test_uncertified_sums(n, late):
    """late: particles behind the loss test's limit, so the moments are swept
    again over the good set they leave"""
    from hpsim_gb300 import HPSim
    for seed in range(3):
        y, phi = _inputs(n, seed)
        odd = np.random.default_rng(seed).choice(np.arange(1, n), 20, replace=False)
        phi[odd[:10]] = 0.99995 * np.pi
        if late:
            phi[odd[10:]] += 4.0 * np.pi
        beam, sc = _beam(n, y, phi)
        HPSim.Simulator(beam, HPSim.BeamLine(elements=_line(1)), sc).simulate()
        assert sc.get_counter("stat_sweeps") == 1
        if late:
            good = y.copy()
            good[odd[10:]] = 0.0
            edge = _edge(_single_block_sum(good), _single_block_sum(good, "fma"), n)
        else:
            g = _blocks(n, 1)
            edge = _edge(_grid_sum(y, g), _grid_sum(y, g, "fma"), n)
        assert _mesh_edge(sc) == edge


@pytest.mark.parametrize("lockstep", [False, True])
def test_sums_in_a_batch(lockstep):
    from hpsim_gb300 import HPSim
    sims, want, scs = [], [], []
    for k, n in enumerate((5001, 40000, 311297)):
        y, phi = _inputs(n, k)
        beam, sc = _beam(n, y, phi)
        g = _blocks(n, 2)
        want.append(_edge(_grid_sum(y, g), _grid_sum(y, g, "mul"), n))
        scs.append(sc)
        sims.append(HPSim.Simulator(beam, HPSim.BeamLine(elements=_line(3)), sc))
    batch = HPSim.Batch(sims)
    batch.set_lockstep(lockstep)
    batch.simulate()
    assert batch.last_mode()[0] == ("lockstep" if lockstep else "graphs")
    assert [_mesh_edge(sc) for sc in scs] == want
