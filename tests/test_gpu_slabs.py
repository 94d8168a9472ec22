"""Cell slabs of the fine grid: a cell's records are skipped only where no
triangle of it can report a hit, so replayed walks equal the oracle's scan of
the reference grid bit for bit -- with cells of one record and of hundreds
(past the count the cell keeps), with several surfaces in a cell, with
needle-shaped triangles, and with vertices outside the box.
"""
import numpy as np
import pytest

import oracle as O
from scenarios import MeshCase, draws

pytestmark = pytest.mark.gpu
F = np.float32


class OddMeshCase(MeshCase):
    """MeshCase plus needles (height 1e-2 to 1e-4 of their length) and a triangle reaching outside the box, written
    to the same kind of file."""

    def __init__(self, tmpdir, membranes, **kw):
        super().__init__(tmpdir, membranes=membranes, **kw)
        from dsim_gb300 import substrates as S
        rng = np.random.default_rng(9)
        V, T, mem, fib = [self.tube[k] for k in ("vertices", "trgls", "membrane", "fiber")]
        n = 120
        a = rng.uniform(-7, 7, (n, 3))
        d = rng.standard_normal((n, 3))
        d /= np.linalg.norm(d, axis=1)[:, None]
        e = np.cross(d, rng.standard_normal((n, 3)))
        e /= np.linalg.norm(e, axis=1)[:, None]
        h = 10.0 ** rng.uniform(-4, -2, (n, 1))
        new = np.stack([a, a + 1.5 * d, a + (0.2 + 0.6 * rng.random((n, 1))) * d + 1.5 * h * e], 1)
        wide = np.array([[[-14, -14, 3.1], [14, -14, 3.2], [0, 15, 3.3]]], float)
        new = np.concatenate([new, wide]).reshape(-1, 3).astype(F)
        k = len(new) // 3
        self.tube = dict(vertices=np.concatenate([V, new]).astype(F),
                         trgls=np.concatenate([T, len(V) + np.arange(3 * k).reshape(k, 3)]).astype(np.uint32),
                         membrane=np.concatenate([mem, np.full(k, 2 if membranes == "G" else 0, np.uint32)]),
                         fiber=np.concatenate([fib, np.zeros(k, np.uint32)]))
        S.write_mesh_file(self.path, self.tube)


@pytest.mark.parametrize("membranes,accel,records", [("G", None, 32), ("AM", None, 32), ("G", 2, 32), ("AM", 5, 64),
                                                     ("G", 30, 16), ("AM", 90, 32), ("G", 190, 64)])
def test_replay_parity_with_odd_triangles(engine, tmp_path, membranes, accel, records):
    _replay_parity(OddMeshCase(tmp_path, membranes, N=1200, permeability=0.05), accel, records)


@pytest.mark.parametrize("membranes,ring,verts", [("G", 0.4, 16), ("AM", 0.2, 24), ("AM", 0.8, 12)])
def test_replay_parity_with_rings_on_cell_faces(engine, tmp_path, membranes, ring, verts):
    """Triangles that end on faces of the reference grid (cells of 0.4 um), whose lists rounding decides: a single hit
    is taken without the walk over the cells only clear of the faces."""
    _replay_parity(MeshCase(tmp_path, membranes=membranes, N=4000, ring=ring, verts=verts), None, 32)


def _replay_parity(case, accel, records, iters=50):
    from dsim_gb300.engine import Mesh, Spins, mesh_params, mesh_run
    d = draws(iters, case.N, seed=3)
    mo = O.Mesh(case.path, case.spaceScale)
    cc, tic, maxtpc = O.populate_cubes(mo.vertices, mo.trgls, 50)
    p = O.params3(case.stdDevs, case.T2, case.permeability, case.dt, 50, maxtpc)
    pos = case.pos.copy(); seed = np.zeros(2 * case.N, np.uint32)
    mag = case.mag.copy(); ph = case.phase.copy(); comp = case.comp.copy(); fib = case.fiber.copy()
    cnt = np.zeros(2 * case.N, np.uint32)
    O.integrate3(p, pos, seed, mag, ph, comp, fib, mo.vertices, mo.helpers, mo.triInfo, cc, tic, case.g, case.pc, iters,
                 draws=d, counts=cnt)
    m = Mesh.load(case.path, case.spaceScale)
    m.set_records(records)
    if accel is not None:
        m.set_accel(accel)
    s = Spins(case.N)
    s.set(case.pos, case.mag, case.phase, case.comp, case.fiber)
    q = mesh_params(case.stdDevs, case.T2, case.permeability, case.dt, case.pc)
    mesh_run(m, s, q, case.g, iterations=iters, draws=d, count=True)
    gp, gm, gph, gc, gf = s.get()
    assert np.array_equal(s.counts().reshape(-1), cnt)
    assert np.array_equal(gp.view(np.uint32), pos.view(np.uint32))
    assert np.array_equal(gm.view(np.uint32), mag.view(np.uint32))
    assert np.array_equal(gph.view(np.uint32), ph.view(np.uint32))
    assert np.array_equal(gc, comp) and np.array_equal(gf, fib)
