"""What a spin object holds on the device, and arrays read into memory that no one
has written yet."""
import numpy as np
import pytest

from scenarios import MeshCase

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("n", [50_000, 300_000])
def test_arrays_pass_through_the_second_set_of_slots(engine, tmp_path, n):
    """Device bytes: 36 a spin at first (seven words of state, two counters), as many words again once arrays came or
    went or a run reordered the spins, and nothing more for the arrays' passage."""
    from dsim_gb300.engine import Mesh, Spins, mesh_params, mesh_run
    case = MeshCase(tmp_path, N=n)
    m = Mesh.load(case.path, case.spaceScale)
    s = Spins(n)
    fixed = 608 * 15 * 8 + 128 + 7 * 4 * 64                  # signal scratch, small words, the slots' rounding
    assert 36 * n <= s.nbytes <= 36 * n + fixed
    s.set(case.pos, case.mag, case.phase, case.comp, case.fiber)
    held = s.nbytes
    assert held <= 64 * n + 2 * fixed
    s.get()
    s.set(case.pos)
    assert s.nbytes == held
    mesh_run(m, s, mesh_params(case.stdDevs, case.T2, case.permeability, case.dt, case.pc), case.g, 3, seed=2)
    assert s.nbytes <= held + 4 * n + 2 * 4 * (2 * 112 ** 3 + 1) + (1 << 16)   # sort keys and their histogram
    s.free()
