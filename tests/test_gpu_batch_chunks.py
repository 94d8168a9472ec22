"""Configured chunks: launches of one to a few steps list their warps otherwise than
long ones, and a batch configured anew between runs lists them anew; a job's spins
depend on neither."""
import numpy as np
import pytest

from scenarios import CylCase, MeshCase
from test_gpu_batch_shapes import _jobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "local", "precise"])
@pytest.mark.parametrize("n", [70, 6000])
def test_jobs_do_not_depend_on_the_chunk(engine, tmp_path, form, n):
    from dsim_gb300.engine import Batch, Cylinders, Mesh
    mc, cc = MeshCase(tmp_path, membranes="AM", N=7000), CylCase(tmp_path, N=7000, inner=0.7)
    m, c = Mesh.load(mc.path, mc.spaceScale), Cylinders.load(cc.path, cc.spaceScale)
    mesh, cyl = _jobs(mc, cc, n, 48, form)
    got = []
    for chunks in ((48,), (1,), (8,), (9,), (2, 16, 1)):
        b = Batch(1 << 15, 4)
        sm, sc = b.add_mesh(m), b.add_cyl(c)
        ids = b.submit(sm, **mesh), b.submit(sc, **cyl)
        for k, chunk in enumerate(chunks):
            b.configure(chunk=chunk, occupancy=(4, 5, 8)[k])
            if k + 1 < len(chunks):
                b.advance(16)
            else:
                b.run()
        assert b.status() == 0
        got.append([([x for i, x in enumerate(b.get(j, n)) if i != 2], b.counts(j),
                     b.get_precise(j, n) if form != "plain" else ()) for j in ids])
        b.close()
    for other in got[1:]:
        for (g0, k0, p0), (g1, k1, p1) in zip(got[0], other):
            assert np.array_equal(k0, k1)
            for a, b_ in zip((*g0, *p0), (*g1, *p1)):
                assert np.array_equal(a, b_)
