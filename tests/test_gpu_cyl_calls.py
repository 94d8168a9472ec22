"""Cylinder runs in calls of any length: a call of a dozen steps or more runs the
spins by region, a shorter one and a free walk in their own order, few spins in
thin warps, many in full ones; no spin's walk depends on it."""
import numpy as np
import pytest

from scenarios import CylCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("perm", [0.02, 1.0])
@pytest.mark.parametrize("n", [1, 3000, 9000, 41_000, 170_001])
def test_walks_do_not_depend_on_the_calls(engine, tmp_path, n, perm):
    from dsim_gb300.engine import Cylinders, Spins, cyl_params, cyl_run
    case = CylCase(tmp_path, N=n, permeability=perm)
    c = Cylinders.load(case.path, case.spaceScale)
    p = cyl_params(2.0, 2.0, 0.2, case.spaceScale, 70.0, 8.0, 80.0, case.permeability, case.inner, case.dt, case.pc)
    xy, r, um = np.asarray(case.xy), np.asarray(case.r), case.pos.reshape(-1, 3)[:, :2].astype(float) * case.spaceScale
    d = np.hypot(um[:, None, 0] - xy[:, 0], um[:, None, 1] - xy[:, 1]) / r
    near, d = d.argmin(1), d.min(1)
    imo = np.where(d < float(case.inner), 0, np.where(d <= 1, 1, 2)).astype(np.uint32)
    walks = []
    for lengths in ([36], [12, 24], [11] * 3 + [3], [1] * 36):
        s = Spins(n)
        s.set_cyl(case.pos, None, None, imo, np.where(imo < 2, near, 0xFFFFFFFF).astype(np.uint32))
        done = 0
        for k in lengths:
            cyl_run(c, s, p, case.g, k, seed=9, step0=done, count=True)
            done += k
        assert s.status() == 0
        walks.append((*s.get_cyl(), s.counts()))
        s.free()
    for other in walks[1:]:
        for a, b in zip(walks[0], other):
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
