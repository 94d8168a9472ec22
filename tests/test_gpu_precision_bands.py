"""Cylinder precision jobs whose every decision is close: spins on the inner and
outer membranes and on the borders of grid cells, to within 1e-8 to 1e-5 of the
box, moving by steps as small.  The FP64 form takes a side of a membrane or a
cell from FP32 where that is certain and from the double value otherwise, so its
walks stay those of the FP64 oracle, bit for bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("D,inner,perm", [(2e-4, 0.7, 0.05), (2e-8, 0.7, 0.05), (2e-8, 1.0, 0.0), (2e-11, 0.7, 0.02)])
def test_spins_on_membranes_and_cell_borders_equal_fp64_oracle(engine, tmp_path, D, inner, perm):
    from dsim_gb300.engine import Batch, Cylinders, phase_constant, pgse_table, rng_draws
    from scenarios import CylCase
    case = CylCase(tmp_path, permeability=perm, inner=inner, N=1500)
    fp, maxR = O.load_fibers2(case.path, case.spaceScale)
    cc, cubes, n, maxfpc, L = O.build_grid2(fp, maxR)
    f = np.asarray(fp).reshape(-1, 4)
    rng = np.random.default_rng(3)
    pos = case.pos.reshape(-1, 3).copy()
    k = rng.integers(0, len(f), case.N)
    r = np.sqrt(f[k, 3].astype(np.float64)) * np.where(rng.random(case.N) < 0.5, 1.0, float(inner))
    r += rng.choice([-1.0, 1.0], case.N) * 10.0 ** rng.uniform(-8, -5, case.N)
    a = rng.uniform(0, 2 * np.pi, case.N)
    axis = np.where(f[k, 0] == 2.0, 0, np.where(f[k, 2] == 2.0, 2, 1))
    for i in range(1000):  # on a membrane of fiber k, exactly to the rounding of float
        u, v = [c for c in range(3) if c != axis[i]]
        p = f[k[i], u] + r[i] * np.cos(a[i]), f[k[i], v] + r[i] * np.sin(a[i])
        if max(abs(p[0]), abs(p[1])) < 0.95:
            pos[i, u], pos[i, v] = p
    for i in range(800, case.N):  # on a border of a cell, or of a fine cell
        c = rng.integers(0, 3)
        pos[i, c] = F(-1.0 + rng.integers(1, 8 * n) * float(L) / 8 + rng.choice([0.0, 1e-8, -1e-7, 1e-6]))
    pos = pos.astype(F).reshape(-1)
    pos4 = np.zeros((case.N, 4), F)
    pos4[:, :3] = pos.reshape(-1, 3)
    near, imo = np.zeros(case.N, np.uint32), np.zeros(case.N, np.uint32)
    O.lib().or2_find_nearest(case.N, pos4.reshape(-1), fp, n, L, maxfpc, cc, cubes, float(inner), near, imo)
    steps, dt, seed = 60, case.dt, 11
    ss = F(case.spaceScale)
    adc = (F(D) / (ss * ss), F(D) / (ss * ss), F(D) / (ss * ss))
    sd = [float(np.sqrt(F(2) * q * F(dt))) for q in adc] + [0.0]
    table = pgse_table(steps, float(dt), 0.3 * steps * float(dt), 0.6 * steps * float(dt))
    c = Cylinders.load(case.path, case.spaceScale)
    b = Batch(1536, 1)
    j = b.submit(b.add_cyl(c), pos, imo.astype(np.uint8), near, precise=True, steps=steps, dt=dt, step_sd=sd,
                 T2=[70.0, 8.0, 80.0, 0.0], phase_constant=phase_constant(42576.0, dt), seed=seed, permeability=perm,
                 waveform="table", table=table, inner_radius_proportion=inner)
    b.run()
    assert b.status() == 0
    gpos, gmag = b.get_precise(j, case.N)
    _, _, _, gimo, _ = b.get(j, case.N)
    P = O.Params2()
    P.intraAdcScaled, P.myelinAdcScaled, P.extraAdcScaled = adc
    P.T2fiber, P.T2myelin, P.T2outside = 70.0, 8.0, 80.0
    P.permeability, P.innerRadiusProportion, P.spinRadius, P.deltaTime = perm, inner, 0.005, float(dt)
    P.numCubes, P.maxFibersPerCube, P.cubeLength = n, maxfpc, L
    d = np.stack([rng_draws(seed, 0, t, case.N) for t in range(steps)])
    rpos, rmag, rimo, rnear = pos.astype(np.float64), np.ones(case.N), imo.copy(), near.copy()
    O.integrate2_f64_multi(P, rpos, rmag, rimo, rnear, fp, cc, cubes, np.zeros((1, 3)), table.astype(np.float64),
                           1.0, d, nthreads=4)
    assert np.array_equal(gpos.reshape(-1).view(np.uint64), rpos.view(np.uint64))
    assert np.array_equal(gmag.view(np.uint64), rmag.view(np.uint64))
    assert np.array_equal(gimo, rimo.astype(np.uint8))
    b.close()
