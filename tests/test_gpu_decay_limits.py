"""T2 values at the ends of their range, in every form of a batch job: magnitudes
follow mag += -mag / T2 * dt in the form's own precision, bit for bit.  An
infinite T2 is no decay (and neither is 0, which means none); a subnormal one
overflows as the division does."""
import numpy as np
import pytest

from scenarios import CylCase, MeshCase

pytestmark = pytest.mark.gpu
F = np.float32
STEPS = 12
VALUES = [np.inf, 0.0, 1e-45, 3e-39, 80.0, 3.4e38]


def _decay(T2, dt, dtype):
    m, T2, dt = dtype(1), dtype(F(T2)), dtype(F(dt))
    with np.errstate(all="ignore"):
        for _ in range(STEPS):
            if T2 > 0:
                m = m + -m / T2 * dt
    return m


@pytest.mark.parametrize("form", ["plain", "local", "precise"])
@pytest.mark.parametrize("kind", ["mesh", "cylinders"])
@pytest.mark.parametrize("T2", VALUES)
def test_magnitudes_at_the_ends_of_T2(engine, tmp_path, kind, form, T2):
    from dsim_gb300.engine import Batch, Cylinders, Mesh
    n = 200
    b = Batch(1 << 12, 2)
    if kind == "mesh":
        case = MeshCase(tmp_path, N=n)
        m = Mesh.load(case.path, case.spaceScale)
        sub, comp, fib, sd = b.add_mesh(m), case.comp, case.fiber.astype(np.uint32), case.stdDevs
    else:
        case = CylCase(tmp_path, N=n)
        c = Cylinders.load(case.path, case.spaceScale)
        sub, comp, fib, sd = b.add_cyl(c), np.full(n, 2, np.uint8), None, [0.01, 0.01, 0.01, 0.0]
    j = b.submit(sub, pos=case.pos, comp=comp, fiber=fib, steps=STEPS, dt=case.dt, step_sd=sd, T2=[T2] * 4,
                 phase_constant=case.pc, seed=5, permeability=0.02, delta=0.04, Delta=0.06, precise=form == "precise",
                 local=form == "local")
    b.run()
    assert b.status() == 0
    want = _decay(T2, case.dt, np.float64 if form == "precise" else F)
    mag = b.get(j, n)[1]
    assert np.array_equal(mag, np.full(n, F(want)), equal_nan=True)
    if form == "precise":
        assert np.array_equal(b.get_precise(j, n)[1], np.full(n, want), equal_nan=True)
    sums = b.signal(j, np.array([[1.0, 2.0, 3.0]], F))
    if np.isinf(T2) or T2 == 0:
        assert want == 1 and np.all(np.isfinite(sums)) and abs(sums[0, 0, 0]) > 0
    b.close()
