"""The compartment search's walk along a line, against ray crossings in double
(numpy): lines along each axis, through grids of one to many cells, from spins in
and outside the box, and lines that cross as many membranes as the search keeps,
and one more (status bit 4).  Spins whose line comes within 1e-4 of an edge or of
its own ends are left out: there the search may tilt the line at random.  Many
spins are searched a thread each, few a warp each: the same spins find the same
either way, tilts included."""
import numpy as np
import pytest

from scenarios import MeshCase

pytestmark = pytest.mark.gpu
F = np.float32
NONE = 0xFFFF


def _expected(V, T, mem, fib, pos, near=1e-4):
    """(compartment, fiber, clear) of every spin; V in normalised float32."""
    V, pos = V.astype(np.float64), pos.astype(np.float64)
    top = np.abs(V).max(0)
    a = np.abs(pos)
    axis = np.where((a[:, 0] > a[:, 1]) & (a[:, 0] > a[:, 2]), 0, np.where(a[:, 1] > a[:, 2], 1, 2))
    p1, u, v = V[T[:, 0]], V[T[:, 1]] - V[T[:, 0]], V[T[:, 2]] - V[T[:, 0]]
    n = np.cross(u, v)
    uu, uv, vv = (u * u).sum(1), (u * v).sum(1), (v * v).sum(1)
    comp, fiber, clear = (np.zeros(len(pos), int) for _ in range(3))
    for i, s in enumerate(pos):
        d = np.zeros(3)
        d[axis[i]] = (1.0 if s[axis[i]] >= 0 else -1.0) * 1.1 * top[axis[i]] - s[axis[i]]
        den = n @ d
        ok = np.abs(den) > 1e-14
        r = np.where(ok, ((p1 - s) * n).sum(1) / np.where(ok, den, 1.0), -9.0)
        w = s + r[:, None] * d - p1
        wu, wv = (w * u).sum(1), (w * v).sum(1)
        D = uv * uv - uu * vv
        b, c = (uv * wv - vv * wu) / D, (uv * wu - uu * wv) / D
        inside = np.minimum(np.minimum(b, c), 1 - b - c)          # > 0 within the triangle
        edge = (np.abs(inside) < near) & (r > -near) & (r < 1 + near)
        ends = (inside > -near) & ((np.abs(r) < near) | (np.abs(r - 1) < near))
        flat = ~ok & (np.abs(((p1 - s) * n).sum(1)) < 1e-6 * np.linalg.norm(n, axis=1))
        clear[i] = not (edge | ends | flat).any()
        hit = (inside > 0) & (r > 0) & (r < 1)
        keys, times = np.unique(fib[hit].astype(np.int64) * 4 + mem[hit], return_counts=True)
        odd = keys[times % 2 == 1]
        fiber[i] = NONE
        for t in range(3):
            of = odd[(odd & 3) == t]
            if len(of):
                comp[i], fiber[i] = (1, 2, 3)[t], of.min() >> 2
                break
    return comp, fiber, clear.astype(bool)


def _search(V, T, mem, fib, pos, nf):
    from dsim_gb300.engine import Mesh, Spins
    m = Mesh.from_arrays(V, T, mem, fib, 1.0)
    m.set_accel(nf)
    s = Spins(len(pos))
    s.set(pos.reshape(-1), None, None, np.full(len(pos), 9, np.uint8), np.full(len(pos), 9, np.uint16))
    moved = m.compartments(s, seed=4)
    _, _, _, comp, fiber = s.get()
    return comp, fiber, moved, s.status()


@pytest.mark.parametrize("axes", [(0, 1, 2), (1, 2, 0), (2, 0, 1)])
@pytest.mark.parametrize("membranes,nf,scale", [("AM", 112, 10.0), ("AM", 1, 10.0), ("G", 2, 10.0), ("G", 33, 6.0),
                                                ("AM", 190, 6.0), ("AM", 5, 12.0)])
def test_lines_along_each_axis(engine, tmp_path, axes, membranes, nf, scale):
    case = MeshCase(tmp_path, membranes=membranes, n_axons=4)
    t = case.tube
    V = (t["vertices"][:, axes] / F(scale)).astype(F)               # at scale 6 the tubes reach 1.33
    rng = np.random.default_rng(nf)
    pos = rng.uniform(-1.0, 1.0, (600, 3)) * (1.6 if scale < 8 else 0.99)
    for i in range(300):                                            # half of them in or near a tube
        k = rng.integers(0, len(t["radii"]))
        (cx, cy), r = t["centres"][k], t["radii"][k]
        a, q = rng.uniform(0, 2 * np.pi), rng.uniform(0, 1.6) * r
        pos[i] = np.array([cx + q * np.cos(a), cy + q * np.sin(a), rng.uniform(-8.5, 8.5)])[list(axes)] / scale
    pos = pos.astype(F)
    want, wfib, clear = _expected(V, t["trgls"], t["membrane"], t["fiber"], pos)
    comp, fiber, moved, status = _search(V, t["trgls"], t["membrane"], t["fiber"], pos, nf)
    assert status == 0 and moved == 0
    assert clear.mean() > 0.9 and len(np.unique(want[clear])) == (3 if membranes == "AM" else 2)
    a = np.abs(pos[clear])
    assert all((a.argmax(1) == k).sum() > 30 for k in range(3))
    assert np.array_equal(comp[clear], want[clear])
    assert np.array_equal(fiber[clear], wfib[clear])


def _shells(count):
    """Boxes about a common centre, box k of half-edge 0.2 + 0.015 k, each a fiber of its own."""
    c = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], float)
    quads = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    tri = np.array([t for a, b, d, e in quads for t in ((a, b, d), (a, d, e))])
    V = np.concatenate([c * (0.2 + 0.015 * k) for k in range(count)])
    T = np.concatenate([tri + 8 * k for k in range(count)])
    return V.astype(F), T.astype(np.uint32), np.full(len(T), 2, np.uint32), np.repeat(np.arange(count), 12).astype(np.uint32)


@pytest.mark.parametrize("nf", [1, 3, 112])
@pytest.mark.parametrize("count", [31, 32, 33, 40])
def test_lines_across_as_many_membranes_as_are_kept(engine, count, nf):
    V, T, mem, fib = _shells(count)
    rng = np.random.default_rng(count)
    depth = rng.integers(0, count + 1, 200)                         # shells that do not hold the spin
    pos = np.empty((200, 3), F)
    for i, k in enumerate(depth):
        p = rng.uniform(-0.08, 0.08, 3)
        p[rng.integers(0, 3)] = rng.choice([-1, 1]) * (0.2 + 0.015 * k - 0.0071)
        pos[i] = p
    want, wfib, clear = _expected(V, T, mem, fib, pos)
    assert clear.mean() > 0.9 and np.array_equal(wfib[clear], np.where(depth < count, depth, NONE)[clear])
    few = count - depth <= 32                                       # membranes left on the line
    comp, fiber, moved, status = _search(V, T, mem, fib, pos[few], nf)
    assert moved == 0 and status == 0
    ok = clear[few]
    assert np.array_equal(comp[ok], want[few][ok]) and np.array_equal(fiber[ok], wfib[few][ok])
    if not few.all():
        assert _search(V, T, mem, fib, pos[~few], nf)[3] & 4


def _all(V, T, mem, fib, pos, nf):
    from dsim_gb300.engine import Mesh, Spins
    m = Mesh.from_arrays(V, T, mem, fib, 1.0)
    m.set_accel(nf)
    s = Spins(len(pos))
    s.set(pos.reshape(-1), None, None, np.full(len(pos), 9, np.uint8), np.full(len(pos), 9, np.uint16))
    m.compartments(s, seed=4)
    p, _, _, comp, fiber = s.get()
    return p.reshape(-1, 3), comp, fiber, s.status()


@pytest.mark.parametrize("membranes,nf,scale", [("AM", 112, 10.0), ("G", 20, 6.0), ("AM", 3, 12.0)])
def test_many_spins_find_what_few_do(engine, tmp_path, membranes, nf, scale):
    case = MeshCase(tmp_path, membranes=membranes, n_axons=4)
    t = case.tube
    V = (t["vertices"] / F(scale)).astype(F)
    rng = np.random.default_rng(nf)
    pos = rng.uniform(-1.2, 1.2, (300_000, 3)).astype(F)            # a thread each: 100,000 and a quarter of the entries
    pos[:500, :2] = np.asarray(t["centres"])[rng.integers(0, 4, 500)] / scale     # on an axis: lines along edges
    pos[:500, 2] = rng.integers(-8, 9, 500) / scale
    few = 1500                                                      # a warp each, at 3 layers of cells too
    many, some = _all(V, t["trgls"], t["membrane"], t["fiber"], pos, nf), _all(V, t["trgls"], t["membrane"], t["fiber"],
                                                                               pos[:few], nf)
    assert many[3] == some[3] == 0
    for a, b in zip(many[:3], some[:3]):
        assert np.array_equal(a[:few].view(np.uint8), b.view(np.uint8))
    assert len(np.unique(some[1])) == (3 if membranes == "AM" else 2)


@pytest.mark.parametrize("count", [32, 33])
def test_many_spins_across_as_many_membranes_as_are_kept(engine, count):
    V, T, mem, fib = _shells(count)
    pos = np.full((150_000, 3), 0.01, F) * np.array([1, -2, 0.5], F)
    comp, fiber, moved, status = _search(V, T, mem, fib, pos, 112)
    assert moved == 0 and status == (4 if count > 32 else 0)
    if count == 32:
        assert np.all(comp == 3) and np.all(fiber == 0)
