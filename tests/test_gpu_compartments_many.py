"""The compartment search over more spins than 2^27, where 32 threads a spin pass
2^32: every spin is examined, and once."""
import numpy as np
import pytest

from scenarios import MeshCase

pytestmark = pytest.mark.gpu
F = np.float32


def test_spins_past_2_27_are_examined(engine, tmp_path):
    from dsim_gb300.engine import Mesh, Spins, check, native
    case = MeshCase(tmp_path, membranes="AM", N=64)
    (cx, cy), r = case.tube["centres"][1], case.tube["radii"][1]
    # off the axis, whose lines meet edges and are tilted at random: one in 10^6 of those meets another
    inside = np.array([cx + 0.0131, cy - 0.0213, 0.137]) / case.spaceScale
    outside = np.array([0.97, -0.96, 0.93])     # no tube reaches it: they end at 0.6 + 1.25 * 1.2 r and at |z| = 0.8
    N = (1 << 27) + 4099
    s = Spins(N)
    pos = np.empty((N, 3), F)
    pos[0::2], pos[1::2] = inside, outside
    check(native().dsim_spins_set(s.h, pos.reshape(-1), None, None, np.full(N, 7, np.uint8), None))
    m = Mesh.load(case.path, case.spaceScale)
    assert m.compartments(s, seed=3) == 0
    assert s.status() == 0
    comp, fib = np.zeros(N, np.uint8), np.zeros(N, np.uint16)
    check(native().dsim_spins_get(s.h, None, None, None, comp, fib))
    assert np.all(comp[0::2] == 1) and np.all(comp[1::2] == 0)
    assert np.all(fib[0::2] == 1) and np.all(fib[1::2] == 0xFFFF)
    m.free(); s.free()
