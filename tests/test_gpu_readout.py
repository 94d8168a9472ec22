"""Readout kernels at the sizes where they branch, against numpy in float64 on
the same spins.

Tolerance: with u = 2^-53 a spin's term is off by at most u (3 |phi| + 4) times
its magnitude on either side (three roundings in the phase, two ulps in the
sine), and a sum of n terms of at most 1 by n u a term."""
import numpy as np
import pytest

from scenarios import CylCase, MeshCase

pytestmark = pytest.mark.gpu
F = np.float32
U = 2.0 ** -53


def _sums(mag, phase, comp):
    out = np.zeros((5, 3))
    for k in range(5):
        on = np.ones(len(mag), bool) if k == 0 else comp == k - 1
        out[k] = (mag * np.cos(phase))[on].sum(), (mag * np.sin(phase))[on].sum(), on.sum()
    return out


def _tol(n, phimax):
    return n * U * (2 * (3 * phimax + 4) + 2 * n)


@pytest.mark.parametrize("n,ng", [(1, 1), (31, 33), (32, 32), (33, 31), (65, 384), (500, 1), (5000, 100)])
@pytest.mark.parametrize("region", [0.0, 0.6])
def test_batch_signal_against_numpy(engine, tmp_path, n, ng, region):
    from dsim_gb300.engine import Batch, Cylinders
    case = CylCase(tmp_path, N=5000)
    c = Cylinders.load(case.path, case.spaceScale)
    imo = (np.arange(n) % 3).astype(np.uint8)
    b = Batch(1 << 13, 2)
    j = b.submit(b.add_cyl(c), case.pos[:3 * n], imo, np.full(n, 5, np.uint32), 20, case.dt, [0.02, 0.01, 0.02],
                 [70.0, 8.0, 80.0], case.pc, 3, permeability=1.0, waveform="table", table=np.ones(20, F))
    b.run()
    pos, mag, mom, comp, _ = b.get(j, n)
    rng = np.random.default_rng(n + ng)
    G = (rng.standard_normal((ng, 3)) * 1e-4 * 10.0 ** rng.uniform(-2, 3, (ng, 1))).astype(F)
    M = mom[:, :3].astype(np.float64) - mom[:, 3:].astype(np.float64)
    keep = np.ones(n, bool) if region == 0 else (np.abs(pos.reshape(-1, 3).astype(np.float64)) < region).all(1)
    got = b.signal(j, G, region)
    for g in range(ng):
        phi = M @ (float(case.pc) * G[g].astype(np.float64))
        want = _sums(mag[keep].astype(np.float64), phi[keep], comp[keep])
        tol = _tol(max(keep.sum(), 1), np.abs(phi).max())
        assert np.array_equal(got[g, :, 2], want[:, 2])
        assert np.abs(got[g] - want).max() <= tol


def test_batch_signal_of_huge_phases_stays_bounded(engine, tmp_path):
    from dsim_gb300.engine import Batch, Cylinders
    case = CylCase(tmp_path, N=100)
    b = Batch(128, 1)
    j = b.submit(b.add_cyl(Cylinders.load(case.path, case.spaceScale)), case.pos, np.full(100, 2, np.uint8), None, 4,
                 case.dt, [0.02] * 3, [0.0] * 3, case.pc, 3, permeability=1.0, waveform="table", table=np.ones(4, F))
    b.run()
    s = b.signal(j, np.array([[1e10, 0, 0], [0, 1e25, 0], [0, 0, 3e38]], F))
    assert (np.hypot(s[:, 0, 0], s[:, 0, 1]) <= 100 * (1 + 1e-12)).all() and (s[:, 0, 2] == 100).all()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 20000, 155648, 155649])
def test_signal_against_numpy(engine, tmp_path, n):
    from dsim_gb300.engine import Spins
    rng = np.random.default_rng(n)
    pos = rng.uniform(-0.99, 0.99, (n, 3)).astype(F)
    mag, ph = rng.random(n, F), (rng.standard_normal(n) * 20).astype(F)
    comp = rng.integers(0, 4, n).astype(np.uint8)
    s = Spins(n)
    s.set(pos, mag, ph, comp, np.zeros(n, np.uint16))
    for region in (0.0, 0.5):
        keep = np.ones(n, bool) if region == 0 else (np.abs(pos.astype(np.float64)) < region).all(1)
        want = _sums(mag[keep].astype(np.float64), ph[keep].astype(np.float64), comp[keep])
        got = s.signal(region)
        assert np.array_equal(got[:, 2], want[:, 2])
        assert np.abs(got - want).max() <= _tol(max(keep.sum(), 1), 100.0)
