"""A signal read after the spins adds them in spin order: it is the signal of the
same arrays given to a new object, to the last bit, however the runs before it
reordered the slots."""
import numpy as np
import pytest

from scenarios import MeshCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [900, 40_000, 170_001])
def test_signal_after_get_is_in_spin_order(engine, tmp_path, n):
    from dsim_gb300.engine import Mesh, Spins, mesh_params, mesh_run
    case = MeshCase(tmp_path, N=n)
    m = Mesh.load(case.path, case.spaceScale)
    s = Spins(n)
    s.set(case.pos, case.mag, case.phase, case.comp, case.fiber)
    p = mesh_params(case.stdDevs, case.T2, case.permeability, case.dt, case.pc)
    for k in range(3):
        mesh_run(m, s, p, case.g, 5, seed=6, step0=5 * k)
        arrays = s.get()
        got = s.signal()
        t = Spins(n)
        t.set(*arrays)
        assert np.array_equal(got.view(np.uint64), t.signal().view(np.uint64))
        t.free()
