"""Spin arrays in and out: one copy for all of them where they are small, a copy
each where they are not, any of them left out, before and after the spins were
reordered by a run.  What is not given stays with its spin; what comes back is in
spin order, byte for byte."""
import numpy as np
import pytest

from scenarios import CylCase, MeshCase

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("n", [1, 33, 11397, 11398, 40000])  # 23 bytes a spin: 256 KB is 11397.6 of them
@pytest.mark.parametrize("walked", [False, True])
def test_mesh_arrays_keep_their_spins(engine, tmp_path, n, walked):
    from dsim_gb300.engine import Mesh, Spins, mesh_params, mesh_run
    case = MeshCase(tmp_path, N=n)
    rng = np.random.default_rng(n)
    want = [case.pos.reshape(-1), rng.random(n, F), rng.random(n, F), rng.integers(0, 4, n).astype(np.uint8),
            rng.integers(0, 60000, n).astype(np.uint16)]
    s = Spins(n)
    s.set(*want)
    if walked:
        m = Mesh.load(case.path, case.spaceScale)
        mesh_run(m, s, mesh_params(case.stdDevs, case.T2, case.permeability, case.dt, case.pc), case.g, 3, seed=2)
        want = list(s.get())
        mesh_run(m, s, mesh_params(case.stdDevs, case.T2, case.permeability, case.dt, case.pc), case.g, 3, seed=2)
        s.set(*want)                                    # given in spin order over reordered slots
    for k in range(5):
        new = [None] * 5
        new[k] = want[k] = np.ascontiguousarray(want[k][::-1])
        if k == 3:
            want[4] = np.full(n, 0xFFFF, np.uint16)     # compartments without fibers: no fiber
        if k == 4:
            want[3] = np.zeros(n, np.uint8)             # fibers without compartments: compartment 0
        s.set(*new)                                     # one array, the others stay
        for a, b in zip(s.get(), want):
            assert np.array_equal(a.view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


@pytest.mark.parametrize("n", [1, 9362, 9363, 30000])       # 28 bytes a spin
def test_cylinder_arrays_keep_their_spins(engine, tmp_path, n):
    from dsim_gb300.engine import Cylinders, Spins, cyl_params, cyl_run
    case = CylCase(tmp_path, N=n)
    rng = np.random.default_rng(n)
    want = [case.pos.reshape(-1), rng.random(n, F), rng.random(n, F), np.full(n, 2, np.uint32),
            rng.integers(0, 64, n).astype(np.uint32)]
    s = Spins(n)
    s.set_cyl(*want)
    for a, b in zip(s.get_cyl(), want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    p = cyl_params(2.0, 2.0, 0.2, case.spaceScale, 70.0, 8.0, 80.0, case.permeability, case.inner, case.dt, case.pc)
    c = Cylinders.load(case.path, case.spaceScale)
    cyl_run(c, s, p, case.g, 4, seed=3)
    after = s.get_cyl()
    t = Spins(n)
    t.set_cyl(*after)
    for a, b in zip(t.get_cyl(), after):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    s.set_cyl(want[0], want[1], want[2])                # regions left out: as the call documents, from the position
    pos, mag, ph, _, _ = s.get_cyl()
    assert np.array_equal(pos, want[0]) and np.array_equal(mag, want[1]) and np.array_equal(ph, want[2])
