"""Cell slabs, lone hits and the triangles' flags in the FP64 and cell-local forms,
whose points come by other ways than the plain form's: among needles, triangles
that end on cell faces and one that leaves the box, the FP64 walk equals the FP64
oracle's at every fine grid, and the cell-local walk does not depend on the grid
(the lists only offer triangles; each is decided by its own records), down to one
cell, whose slab holds every triangle."""
import numpy as np
import pytest

from scenarios import MeshCase
from test_gpu_slabs import OddMeshCase

pytestmark = pytest.mark.gpu
F = np.float32
GRIDS = [(1, 32), (5, 64), (30, 32), (112, 32), (190, 64)]


def _case(tmp_path, kind):
    if kind == "odd AM":
        return OddMeshCase(tmp_path, "AM", N=700, permeability=0.05)
    if kind == "odd G":
        return OddMeshCase(tmp_path, "G", N=700, permeability=0.05)
    return MeshCase(tmp_path, membranes="AM", N=700, ring=0.4, verts=16)


def _walks(case, form, steps, seed=17):
    from dsim_gb300.engine import Batch, Mesh
    m = Mesh.load(case.path, case.spaceScale)
    for nf, records in GRIDS:
        m.set_records(records)
        m.set_accel(nf)
        b = Batch(1 << 10, 1)
        j = b.submit(b.add_mesh(m), pos=case.pos, comp=case.comp, fiber=case.fiber.astype(np.uint32), steps=steps,
                     dt=case.dt, step_sd=case.stdDevs, T2=case.T2, phase_constant=case.pc, seed=seed,
                     permeability=case.permeability, waveform="table", table=np.ones(steps, F),
                     precise=form == "precise", local=form == "local")
        b.run()
        assert b.status() == 0
        pos, mag = b.get_precise(j, case.N)
        _, _, _, comp, fib = b.get(j, case.N)
        yield pos, mag, comp, fib, b.counts(j)
        b.close()


@pytest.mark.parametrize("kind", ["odd AM", "odd G", "rings on faces"])
def test_fp64_walks_equal_the_fp64_oracle(engine, tmp_path, kind):
    from test_gpu_precision import _oracle
    case, steps = _case(tmp_path, kind), 60
    pos64, mag64, comp, fib, cnt, _ = _oracle(case, steps, 17, np.ones((1, steps), F))
    assert cnt.sum() > 500
    for gpos, gmag, gcomp, gfib, gcnt in _walks(case, "precise", steps):
        assert np.array_equal(gcnt, cnt.astype(np.uint64))
        assert np.array_equal(gpos.view(np.uint64), pos64.view(np.uint64))
        assert np.array_equal(gmag.view(np.uint64), mag64.view(np.uint64))
        assert np.array_equal(gcomp, comp) and np.array_equal(gfib & 0xFFFF, fib.astype(np.uint32))


@pytest.mark.parametrize("kind", ["odd AM", "odd G", "rings on faces"])
def test_local_walks_do_not_depend_on_the_fine_grid(engine, tmp_path, kind):
    walks = list(_walks(_case(tmp_path, kind), "local", 60))
    assert walks[0][4].sum() > 500
    for other in walks[1:]:
        for a, b in zip(walks[0], other):
            assert np.array_equal(np.asarray(a).view(np.uint8), np.asarray(b).view(np.uint8))
