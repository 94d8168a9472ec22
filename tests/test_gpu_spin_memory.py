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


@pytest.mark.parametrize("n", [11_500, 300_007])             # either side of one copy for all arrays
@pytest.mark.parametrize("nudge", [0, 4, 4092])
def test_arrays_read_into_fresh_memory_leave_the_rest(engine, n, nudge):
    """Arrays inside one fresh mapping, at odd places of its pages: theirs are written, the words around are not."""
    import ctypes as C
    import mmap
    from dsim_gb300.engine import Spins, check, native
    rng = np.random.default_rng(n)
    want = [rng.random(3 * n, F), rng.random(n, F), rng.random(n, F), rng.integers(0, 4, n).astype(np.uint8),
            rng.integers(0, 60000, n).astype(np.uint16)]
    s = Spins(n)
    s.set(*want)
    raw = mmap.mmap(-1, sum(a.nbytes for a in want) + 6 * 8192)
    whole = np.frombuffer(raw, np.uint8)
    at, out, used = 4096 + nudge, [], np.zeros(len(whole), bool)
    for a in want:
        out.append(whole[at:at + a.nbytes].view(a.dtype))
        used[at:at + a.nbytes] = True
        at += (a.nbytes + 7) // 8 * 8 + 64
    whole[:8] = 7
    check(native().dsim_spins_get(s.h, *out))
    for a, b in zip(out, want):
        assert np.array_equal(a, b)
    rest = whole[~used]
    assert np.all(rest[:8] == 7) and not rest[8:].any()
    s.free()
