"""Reference grids of more than 512 cells per axis (up to 1024 are accepted): a
walk between two flat membranes meets one triangle at a time, so it is the same
whatever the grid's cells are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32
PLANES = (-0.6037, 0.5037)


def _planes(k=40, half=0.999):
    """Squares of 2 half x 2 half at each z of PLANES, k x k x 2 triangles each."""
    x = np.linspace(-half, half, k + 1)
    V, T = [], []
    i, j = (a.reshape(-1) for a in np.meshgrid(np.arange(k), np.arange(k), indexing="ij"))
    for p, z in enumerate(PLANES):
        gx, gy = np.meshgrid(x, x, indexing="ij")
        V.append(np.stack([gx.reshape(-1), gy.reshape(-1), np.full((k + 1) ** 2, z)], 1))
        a = p * (k + 1) ** 2 + i * (k + 1) + j
        T += [np.stack([a, a + k + 1, a + 1], 1), np.stack([a + 1, a + k + 1, a + k + 2], 1)]
    return np.concatenate(V).astype(F), np.concatenate(T).astype(np.uint32)


def _walk(cubes, pos, steps=60):
    from dsim_gb300.engine import Mesh, Spins, mesh_params, mesh_run
    V, T = _planes()
    m = Mesh.from_arrays(V, T, np.full(len(T), 2, np.uint32), np.zeros(len(T), np.uint32), 1.0, numCubes=cubes)
    s = Spins(len(pos))
    s.set(pos.reshape(-1), np.ones(len(pos), F), np.zeros(len(pos), F), np.zeros(len(pos), np.uint8),
          np.full(len(pos), 0xFFFF, np.uint16))
    mesh_run(m, s, mesh_params([0.01] * 4, [80.0] * 4, 0.0, 0.01, 1.0), (1.0, 2.0, 3.0), steps, seed=4, count=True)
    assert s.status() == 0
    out = s.get(), s.counts()
    m.free(); s.free()
    return out


@pytest.mark.parametrize("cubes", [512, 513, 600, 1024])
def test_walks_do_not_depend_on_the_cells(engine, cubes):
    rng = np.random.default_rng(8)
    pos = rng.uniform(-0.95, 0.95, (3000, 3)).astype(F)
    pos[1000:2000, 2] = PLANES[1] + rng.choice([-1, 1], 1000) * rng.uniform(1e-3, 2e-2, 1000)
    pos[2000:, 2] = PLANES[0] + rng.choice([-1, 1], 1000) * rng.uniform(1e-3, 2e-2, 1000)
    got, counts = _walk(cubes, pos)
    want, wcounts = _walk(50, pos)
    assert counts[:, 0].sum() > 1000 and np.array_equal(counts, wcounts)
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
