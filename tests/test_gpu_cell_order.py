"""Cells of the reference grid with more triangles than the sort's shared memory
holds: their lists ascend, whatever the order in which they were filled."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("count", [511, 512, 513, 1024, 1025, 4097, 60_001])
def test_a_cell_of_many_triangles_ascends(engine, count):
    from dsim_gb300.engine import Mesh
    rng = np.random.default_rng(count)
    V = (rng.uniform(-0.9, 0.9, (count, 1, 3)) + rng.uniform(-0.02, 0.02, (count, 3, 3))).astype(F)
    m = Mesh.from_arrays(V.reshape(-1, 3), np.arange(3 * count, dtype=np.uint32).reshape(-1, 3),
                         np.zeros(count, np.uint32), np.zeros(count, np.uint32), 1.0, numCubes=1)
    start, tri = m.grid()
    assert list(start) == [0, count] and m.max_per_cell == count
    assert np.array_equal(tri, np.arange(count, dtype=np.uint32))
    m.free()
