"""Substrate build kernels at the sizes where they branch.

* The reference grid's lists against the oracle's populateCubes for grids
  whose fullest cell holds few, several hundred and more than 512 triangles
  (the last are sorted by a single lane).
* The fine grid's entry count against the separating axes evaluated in double
  on the same float inputs (numpy): the FP32 axes in front of them decide no
  cell differently.
"""
import numpy as np
import pytest

import oracle as O
from scenarios import MeshCase

pytestmark = pytest.mark.gpu
F = np.float32
EPS = float(F(1e-5))


@pytest.mark.parametrize("cubes", [1, 2, 3, 9, 50])
def test_cell_lists_ascend_at_every_cell_size(engine, tmp_path, cubes):
    from dsim_gb300.engine import Mesh
    case = MeshCase(tmp_path, membranes="AM", n_axons=3)
    m = Mesh.load(case.path, case.spaceScale, numCubes=cubes)
    mo = O.Mesh(case.path, case.spaceScale)
    cc, tic, maxtpc = O.populate_cubes(mo.vertices, mo.trgls, cubes)
    start, tri = m.grid()
    assert np.array_equal(np.diff(start.astype(np.int64)), cc.astype(np.int64))
    assert m.max_per_cell == maxtpc and (cubes > 1 or maxtpc > 512)
    dense = tic.reshape(-1, maxtpc)
    for c in np.nonzero(cc)[0]:
        assert np.array_equal(tri[start[c]:start[c + 1]], dense[c, :cc[c]])


def _entries64(V, T, nf):
    """Fine-grid entries by the FP64 axes: for each cell of a triangle's widened bounding box, the triangle's plane and
    the nine edge axes against the cell widened by EPS (outermost cells open outward); a one-cell box needs no test."""
    p = V[T.astype(np.int64)]
    p1, u, v = p[:, 0], p[:, 2] - p[:, 0], p[:, 1] - p[:, 0]          # float32, as the records keep them
    c = np.stack([p1, p1 + v, p1 + u], 1)
    inv = F(nf) / F(2)
    lo = np.clip(np.floor((c.min(1) - F(EPS) + F(1)) * inv), 0, nf - 1).astype(np.int64)
    hi = np.clip(np.floor((c.max(1) + F(EPS) + F(1)) * inv), 0, nf - 1).astype(np.int64)
    total = 0
    for t in range(len(T)):
        ax = [np.arange(lo[t, k], hi[t, k] + 1) for k in range(3)]
        cells = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
        if len(cells) == 1:
            total += 1
            continue
        L = 2.0 / nf
        b0 = np.where(cells == 0, -1e6, -1.0 + cells * L - EPS)
        b1 = np.where(cells == nf - 1, 1e6, -1.0 + (cells + 1) * L + EPS)
        ctr, h = 0.5 * (b0 + b1), 0.5 * (b1 - b0)
        w = c[t].astype(np.float64)[None] - ctr[:, None]
        e = [w[:, 1] - w[:, 0], w[:, 2] - w[:, 1], w[:, 0] - w[:, 2]]
        ok = np.ones(len(cells), bool)
        for i in range(3):
            for j in range(3):
                a = np.zeros((len(cells), 3))
                a[:, (i + 1) % 3], a[:, (i + 2) % 3] = -e[j][:, (i + 2) % 3], e[j][:, (i + 1) % 3]
                q = np.einsum("nk,nck->nc", a, w)
                r = (h * np.abs(a)).sum(1)
                ok &= ~((q.min(1) > r) | (q.max(1) < -r))
        n = np.cross(e[0], e[1])
        ok &= np.abs((n * w[:, 0]).sum(1)) <= (h * np.abs(n)).sum(1)
        total += int(ok.sum())
    return total


@pytest.mark.parametrize("nf", [1, 7, 40, 112])
def test_fine_grid_entries_equal_the_fp64_axes(engine, tmp_path, nf):
    from dsim_gb300.engine import Mesh
    case = MeshCase(tmp_path, membranes="G", n_axons=2)
    m = Mesh.load(case.path, case.spaceScale)
    m.set_accel(nf)
    mo = O.Mesh(case.path, case.spaceScale)
    V = np.asarray(mo.vertices, F).reshape(-1, 3)
    T = np.asarray(mo.trgls).reshape(-1, 3)
    assert m.accel_info()["entries"] == _entries64(V, T, nf)


@pytest.mark.parametrize("size,nf", [(0.02, 64), (0.055, 64), (0.12, 64), (0.3, 64), (0.7, 9)])
def test_fine_grid_entries_of_triangles_of_few_and_many_cells(engine, size, nf):
    """Triangles whose ranges hold from one cell to hundreds (the fill reads the count's bits up to 64 cells and tests
    the cells of larger ones again): entries as the FP64 axes have them, and both passes agree (the sums are the lists')."""
    from dsim_gb300.engine import Mesh
    rng = np.random.default_rng(int(size * 1000))
    T = 400
    ctr = rng.uniform(-0.9, 0.9, (T, 1, 3))
    V = np.clip(ctr + rng.uniform(-size / 2, size / 2, (T, 3, 3)), -0.99, 0.99).astype(F).reshape(-1, 3)
    tri = np.arange(3 * T, dtype=np.uint32).reshape(-1, 3)
    m = Mesh.from_arrays(V, tri, np.zeros(T, np.uint32), np.zeros(T, np.uint32), 1.0, numCubes=8)
    m.set_accel(nf)
    assert m.accel_info()["entries"] == _entries64(V, tri, nf)
    lists = m.grid()
    cc, tic, maxtpc = O.populate_cubes(V.reshape(-1), tri.reshape(-1), 8)
    assert np.array_equal(np.diff(lists[0].astype(np.int64)), cc.astype(np.int64))
    dense = tic.reshape(-1, maxtpc)
    for c in np.nonzero(cc)[0]:
        assert np.array_equal(lists[1][lists[0][c]:lists[0][c + 1]], dense[c, :cc[c]])
