"""Launch shapes: with few spins a warp advances fewer than 32 of them, and the
mesh step picks its blocks per SM by the count.  The spins' walks do not depend
on either: the first n of a large set equal, bit for bit, a set of those n
alone, at counts around the changes of the rules (152 SMs x 20 or 24 warps for
meshes, then 4 to 7 blocks of 128 per SM; x 33 warps for cylinders), and whatever
warp they are dealt to."""
import numpy as np
import pytest

from scenarios import CylCase, MeshCase

pytestmark = pytest.mark.gpu
F = np.float32
STEPS = 25


def _mesh(case, m, n):
    from dsim_gb300.engine import Spins, mesh_params, mesh_run
    s = Spins(n)
    s.set(case.pos[:3 * n], case.mag[:n], case.phase[:n], case.comp[:n], case.fiber[:n])
    mesh_run(m, s, mesh_params(case.stdDevs, case.T2, case.permeability, case.dt, case.pc), case.g, STEPS, seed=5, count=True)
    return (*s.get(), s.counts())


@pytest.mark.parametrize("n", [1, 31, 2433, 3041, 4865, 40961, 58367, 58368, 77825, 97281, 116737, 136193])
def test_mesh_walks_do_not_depend_on_spins_per_warp(engine, tmp_path, n):
    from dsim_gb300.engine import Mesh
    case = MeshCase(tmp_path, membranes="AM", N=165001)
    m = Mesh.load(case.path, case.spaceScale)
    one, all_ = _mesh(case, m, n), _mesh(case, m, case.N)
    for a, b in zip(one, all_):
        k = len(a) // n
        assert np.array_equal(a, b[:n] if a.ndim == 2 else b[:k * n])


@pytest.mark.parametrize("n", [1, 31, 5016, 5017, 10033, 20065, 40129, 80257])
def test_cylinder_walks_do_not_depend_on_spins_per_warp(engine, tmp_path, n):
    from dsim_gb300.engine import Cylinders, Spins, cyl_params, cyl_run
    case = CylCase(tmp_path, N=161000)
    c = Cylinders.load(case.path, case.spaceScale)
    imo = np.full(case.N, 2, np.uint32)
    p = cyl_params(2.0, 2.0, 0.2, case.spaceScale, 70.0, 8.0, 80.0, case.permeability, case.inner, case.dt, case.pc)

    def run(k):
        s = Spins(k)
        s.set_cyl(case.pos[:3 * k], None, None, imo[:k], None)
        cyl_run(c, s, p, case.g, STEPS, seed=5, count=True)
        return (*s.get_cyl(), s.counts())

    one, all_ = run(n), run(case.N)
    for a, b in zip(one, all_):
        k = len(a) // n
        assert np.array_equal(a, b[:n] if a.ndim == 2 else b[:k * n])
