"""libdsim3 calls a host can make between two good ones: a grid whose counters or
entries are out of range is refused before any kernel takes its words for
triangles, and the next call on a good grid walks as the oracle does; calls of
different spin counts keep the plug-in's buffers at the largest one's; a cell edge
of the host's own is taken as it is."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from scenarios import MeshCase, draws

pytestmark = pytest.mark.gpu
F = np.float32
CUBES = 50
SPIN = np.dtype([("mag", "<f4"), ("phase", "<f4"), ("comp", "u1"), ("pad", "u1"), ("fiber", "<u2")])


class Host:
    """A dSim3 host's device arrays and constants for one MeshCase."""

    def __init__(self, case):
        from dsim_gb300 import _lib
        self.L, self.case, self.bases, self.Float3 = _lib.abi3(), case, [], _lib.Float3
        self.mo = O.Mesh(case.path, case.spaceScale)
        self.cc, tic, self.W = O.populate_cubes(self.mo.vertices, self.mo.trgls, CUBES)
        self.tic = np.ascontiguousarray(tic).reshape(-1)
        L, mo = self.L, self.mo
        self.nT = len(mo.triInfo) // 3
        self.dV, self.dH, self.dTI = self.put(mo.vertices), self.put(mo.helpers), self.put(mo.triInfo)
        self.dTic, self.dCc = self.put(self.tic), self.put(self.cc)
        L.bindVertices(self.dV, len(mo.vertices))
        L.bindTriangleHelpers(self.dH, len(mo.helpers))
        L.bindTriInfo(self.dTI, len(mo.triInfo))
        for name, val, ty in (("k_numCubes", CUBES, np.uint32), ("k_totalNumCubes", CUBES ** 3, np.uint32),
                              ("k_maxTrianglesPerCube", self.W, np.uint32), ("k_cubeLength", F(2.0) / F(CUBES), F),
                              ("k_reflectionType", 1, np.uint32), ("k_permeability", case.permeability, F),
                              ("k_deltaTime", case.dt, F)):
            self.constant(name, val, ty)
        for name, tab in (("k_T2Values", case.T2), ("k_stdDevs", case.stdDevs)):
            a = np.ascontiguousarray(tab, F)
            L.copyConstantToDevice(name.encode(), a.ctypes.data, 0, 16)

    def constant(self, name, val, ty):
        a = np.array([val], ty)
        self.L.copyConstantToDevice(name.encode(), a.ctypes.data, 0, 4)

    def put(self, arr):
        arr = np.ascontiguousarray(arr)
        q = C.c_void_p()
        self.L.allocateArray(C.byref(q), max(arr.nbytes, 16))
        self.bases.append(q)
        self.L.copyArrayToDevice(q, arr.ctypes.data, 0, arr.nbytes)
        return q

    def write(self, dst, arr):
        self.L.copyArrayToDevice(dst, arr.ctypes.data, 0, arr.nbytes)

    def spins(self, N):
        """The first N spins of the case, on the device."""
        c = self.case
        s = np.zeros(N, SPIN)
        s["mag"], s["phase"], s["comp"], s["fiber"] = c.mag[:N], c.phase[:N], c.comp[:N], c.fiber[:N]
        return self.put(c.pos[:3 * N]), self.put(np.zeros(2 * N, np.uint32)), self.put(s)

    def step(self, dev, N, d):
        """One call of integrateSystem replaying d [iterations][N][4]; the status it left."""
        return self.call(dev, N, self.put(np.ascontiguousarray(d).reshape(-1)), len(d))

    def call(self, dev, N, draws, iterations):
        c = self.case
        self.L.dsim3_set_replay(draws, None)
        self.L.integrateSystem(*dev, float(c.dt), float(c.permeability), N, self.Float3(*[float(x) for x in c.g]),
                               float(c.pc), iterations, self.dTic, self.dCc)
        return self.L.dsim3_last_status()

    def read(self, dev, N):
        pos, s = np.zeros(3 * N, F), np.zeros(N, SPIN)
        self.L.copyArrayFromDevice(pos.ctypes.data, dev[0], 0, pos.nbytes)
        self.L.copyArrayFromDevice(s.ctypes.data, dev[2], 0, s.nbytes)
        return pos, s

    def oracle(self, N, d, edge=F(2.0) / F(CUBES)):
        c, mo = self.case, self.mo
        p = O.params3(c.stdDevs, c.T2, c.permeability, c.dt, CUBES, self.W)
        p.cubeLength = edge
        pos, mag, ph = c.pos[:3 * N].copy(), c.mag[:N].copy(), c.phase[:N].copy()
        comp, fib = c.comp[:N].copy(), c.fiber[:N].copy()
        capped, _ = O.integrate3(p, pos, np.zeros(2 * N, np.uint32), mag, ph, comp, fib, mo.vertices, mo.helpers,
                                 mo.triInfo, self.cc, self.tic, c.g, c.pc, len(d), draws=d)
        assert capped == 0
        return pos, mag, ph, comp, fib

    def close(self):
        self.L.dsim3_set_replay(None, None)
        self.L.unbindVertices(); self.L.unbindTriangleHelpers(); self.L.unbindTriInfo()
        for q in self.bases:
            self.L.freeArray(q)


@pytest.fixture
def host(engine, tmp_path):
    h = Host(MeshCase(tmp_path, membranes="AM", N=1200))
    yield h
    h.close()


def _equal(got, want):
    pos, s = got
    rpos, mag, ph, comp, fib = want
    assert np.array_equal(pos.view(np.uint32), rpos.view(np.uint32))
    assert np.array_equal(s["mag"].view(np.uint32), mag.view(np.uint32))
    assert np.array_equal(s["phase"].view(np.uint32), ph.view(np.uint32))
    assert np.array_equal(s["comp"], comp) and np.array_equal(s["fiber"], fib)


@pytest.mark.parametrize("fault", ["count", "all counts", "sum past 2^32", "triangle"])
def test_grid_out_of_range_is_refused(host, fault):
    N, full = host.case.N, int(np.argmax(host.cc))
    d = draws(20, N, seed=31)
    cc, tic = host.cc.copy(), host.tic.copy()
    if fault == "count":
        cc[full] = host.W + 1
    elif fault == "all counts":
        cc[:] = host.W + 3
    elif fault == "sum past 2^32":
        cc[7] = 0xFFFFFF00
    else:
        tic[full * host.W] = host.nT
    dev = host.spins(N)
    before = host.read(dev, N)
    host.write(host.dCc, cc)
    host.write(host.dTic, tic)
    assert host.step(dev, N, d) == -4
    assert b"k_maxTrianglesPerCube" in host.L.dsim3_last_error()
    for a, b in zip(host.read(dev, N), before):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))  # no step was taken
    host.L.dsim3_status()
    host.write(host.dCc, host.cc)
    host.write(host.dTic, host.tic)
    assert host.step(dev, N, d) == 0, host.L.dsim3_last_error()
    _equal(host.read(dev, N), host.oracle(N, d))


def _free_bytes():
    free, total = C.c_size_t(), C.c_size_t()
    assert C.CDLL("libcuda.so.1").cuMemGetInfo_v2(C.byref(free), C.byref(total)) == 0
    return free.value


def test_calls_of_different_spin_counts(engine, tmp_path):
    """Two systems in turn: after the larger one's first call no call changes the free memory, and each walks as alone."""
    big, small, its = 720_000, 9000, 3
    h = Host(MeshCase(tmp_path, membranes="AM", N=big))
    try:
        d = draws(its, big, seed=33)
        dB, dS = h.put(d.reshape(-1)), h.put(np.ascontiguousarray(d[:, :small]).reshape(-1))
        devs = [h.spins(n) for n in (big, small, big, small)]
        assert h.call(devs[0], big, dB, its) == 0, h.L.dsim3_last_error()
        h.L.threadSync()
        free = [_free_bytes()]
        for dev, n, dd in ((devs[1], small, dS), (devs[2], big, dB), (devs[3], small, dS)):
            assert h.call(dev, n, dd, its) == 0, h.L.dsim3_last_error()
            h.L.threadSync()
            free.append(_free_bytes())
        assert free == [free[0]] * 4
        want = h.oracle(small, np.ascontiguousarray(d[:, :small]))
        for dev in devs:
            _equal(h.read(dev, small), want)
    finally:
        h.close()


@pytest.mark.parametrize("scale", [1.0 + 1e-7, 1.0 + 1e-5, 1.001, 0.99, 1.3])
def test_cell_edge_of_the_hosts_own(host, scale):
    """k_cubeLength other than the box's 2 / k_numCubes: the reference's walk then visits cells that need not list the
    triangles inside them, and a hit of such a triangle does not count.  Between two calls with the box's own edge."""
    N, own = host.case.N, F(2.0) / F(CUBES)
    d = draws(40, N, seed=35)
    want = {}
    for edge in (own, F(float(own) * scale), own):
        host.constant("k_cubeLength", edge, F)
        dev = host.spins(N)
        assert host.step(dev, N, d) == 0, host.L.dsim3_last_error()
        want[edge] = want[edge] if edge in want else host.oracle(N, d, edge)
        _equal(host.read(dev, N), want[edge])
