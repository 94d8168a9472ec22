"""Launch shapes of a batch: warps of fewer than 32 spins when a kind of job
does not fill the chip, launches of up to 1000 steps when the caller left the
chunk to the batch, warps listed again as jobs finish.  A job's spins do not
depend on any of it: the same jobs in a batch left to itself, in one with short
configured chunks, and beside jobs of other kinds that end earlier give the
same positions, magnitudes, regions and counts (moments of the FP64 form are
kept between launches as float pairs: 2^-46 of the largest)."""
import numpy as np
import pytest

from scenarios import CylCase, MeshCase

pytestmark = pytest.mark.gpu
F = np.float32


def _jobs(mc, cc, n, steps, form):
    kw = dict(precise=form == "precise", local=form == "local")
    ss = F(cc.spaceScale)
    sd = [float(np.sqrt(F(2) * (F(adc) / (ss * ss)) * F(cc.dt))) for adc in (2.0, 0.2, 2.0)] + [0.0]
    mesh = dict(pos=mc.pos[:3 * n], comp=mc.comp[:n], fiber=mc.fiber[:n].astype(np.uint32), dt=mc.dt,
                step_sd=mc.stdDevs, T2=mc.T2, phase_constant=mc.pc, seed=21, permeability=mc.permeability,
                delta=0.2, Delta=0.3, steps=steps, **kw)
    cyl = dict(pos=cc.pos[:3 * n], comp=np.full(n, 2, np.uint8), fiber=None, dt=cc.dt, step_sd=sd,
               T2=[70.0, 8.0, 80.0, 0.0], phase_constant=cc.pc, seed=22, permeability=0.02, delta=0.2, Delta=0.3,
               inner_radius_proportion=0.7, steps=steps, **kw)
    return mesh, cyl


@pytest.mark.parametrize("form", ["plain", "local", "precise"])
@pytest.mark.parametrize("n", [1, 33, 1217, 2500, 7000])
def test_jobs_do_not_depend_on_launch_shapes(engine, tmp_path, form, n):
    from dsim_gb300.engine import Batch, Cylinders, Mesh
    mc, cc = MeshCase(tmp_path, membranes="AM", N=7000), CylCase(tmp_path, N=7000, inner=0.7)
    m, c = Mesh.load(mc.path, mc.spaceScale), Cylinders.load(cc.path, cc.spaceScale)
    mesh, cyl = _jobs(mc, cc, n, 130, form)
    small, _ = _jobs(mc, cc, 500, 105, "plain")
    got = []
    for shape in ("own", "short", "mixed"):
        b = Batch(1 << 16, 8)
        if shape == "short":
            b.configure(chunk=13, graph_chunks=2)
        sm, sc = b.add_mesh(m), b.add_cyl(c)
        if shape == "mixed":
            b.submit(sm, **small)
        ids = b.submit(sm, **mesh), b.submit(sc, **cyl)
        b.run()
        assert b.status() == 0
        got.append([(b.get(j, n), b.counts(j), b.get_precise(j, n) if form != "plain" else ()) for j in ids])
        b.close()
    for other in got[1:]:
        for (g0, k0, p0), (g1, k1, p1) in zip(got[0], other):
            assert np.array_equal(k0, k1)
            for i, (a, b_) in enumerate(zip(g0, g1)):
                if i == 2 and form == "precise":
                    M0, M1 = (x[:, :3].astype(np.float64) - x[:, 3:].astype(np.float64) for x in (a, b_))
                    assert np.abs(M0 - M1).max() <= 12 * 2.0 ** -46 * max(np.abs(M0).max(), 1.0)
                else:
                    assert np.array_equal(a, b_)
            for a, b_ in zip(p0, p1):
                assert np.array_equal(a, b_)


@pytest.mark.parametrize("form", ["plain", "local", "precise"])
def test_full_warps_walk_as_thin_ones(engine, tmp_path, form):
    """A mesh job large enough for 32 spins a warp in every form, against its first spins alone (thin warps)."""
    from dsim_gb300.engine import Batch, Mesh
    mc, cc = MeshCase(tmp_path, membranes="AM", N=99000), CylCase(tmp_path, N=10)
    m = Mesh.load(mc.path, mc.spaceScale)
    out = []
    for n in (mc.N, 1000):
        b = Batch(1 << 17, 1)
        j = b.submit(b.add_mesh(m), **_jobs(mc, cc, n, 30, form)[0])
        b.run()
        assert b.status() == 0
        out.append((*b.get(j, n), *(b.get_precise(j, n) if form != "plain" else ())))
        b.close()
    for a, b_ in zip(*out):
        a, b_ = np.asarray(a), np.asarray(b_)
        assert np.array_equal(a.reshape(mc.N, -1)[:1000], b_.reshape(1000, -1))
