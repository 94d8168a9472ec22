"""libdsim3 on arrays bound at any word of an allocation, with helpers whose vv is
not v . v to the last bit, rewritten in place between two calls: the drop-in reads
the helpers as they are (vv is looked up only where it differs from v . v) and
notices the new contents at every alignment (the hash takes 16 B at a time and the
words at both ends alone), bit for bit with the oracle on the same arrays."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from scenarios import MeshCase, draws

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("words,nudge", [(0, 1), (1, -1), (2, 3), (3, 0)])
def test_arrays_at_any_word_with_their_own_helpers(engine, tmp_path, words, nudge):
    from dsim_gb300 import _lib, substrates as S
    L = _lib.abi3()
    case = MeshCase(tmp_path, membranes="AM", permeability=0.05, N=1200)
    tube2 = dict(case.tube)
    tube2["vertices"] = (case.tube["vertices"] + np.array([0.5, 0.3, -0.25], F)).astype(F)
    path2 = str(tmp_path / "shifted.txt")
    S.write_mesh_file(path2, tube2)
    meshes = []
    for path in (case.path, path2):
        mo = O.Mesh(path, case.spaceScale)
        H = np.array(mo.helpers, F).reshape(-1, 12)
        H[::2, 11] = (H[::2, 11].view(np.int32) + np.int32(nudge)).view(F)   # every other triangle's vv, by ulps
        cc, tic, maxtpc = O.populate_cubes(mo.vertices, mo.trgls, 50)
        meshes.append((mo, np.ascontiguousarray(H.reshape(-1)), cc, tic.reshape(-1, maxtpc), maxtpc))
    W = max(m[4] for m in meshes)
    dense = []
    for m in meshes:
        t = np.zeros((50 ** 3, W), np.uint32)
        t[:, :m[4]] = m[3]
        dense.append(np.ascontiguousarray(t.reshape(-1)))
    its = 30
    d = draws(2 * its, case.N, seed=29)
    p = O.params3(case.stdDevs, case.T2, case.permeability, case.dt, 50, W)
    rpos, seed = case.pos.copy(), np.zeros(2 * case.N, np.uint32)
    mag, ph, comp, fib = case.mag.copy(), case.phase.copy(), case.comp.copy(), case.fiber.copy()
    for k in range(2):
        mo, H, cc = meshes[k][:3]
        capped, _ = O.integrate3(p, rpos, seed, mag, ph, comp, fib, mo.vertices, H, mo.triInfo, cc, dense[k], case.g,
                                 case.pc, its, draws=d[k * its:(k + 1) * its])
        assert capped == 0
    bases = []

    def dev(arr, off=words):
        arr = np.ascontiguousarray(arr)
        q = C.c_void_p()
        L.allocateArray(C.byref(q), arr.nbytes + 16)
        bases.append(C.c_void_p(q.value))
        at = C.c_void_p(q.value + 4 * off)
        L.copyArrayToDevice(at, arr.ctypes.data, 0, arr.nbytes)
        return at

    try:
        mo, H, cc = meshes[0][:3]
        dV, dH, dTI, dTic, dCc = dev(mo.vertices), dev(H), dev(mo.triInfo), dev(dense[0]), dev(cc)
        L.bindVertices(dV, len(mo.vertices))
        L.bindTriangleHelpers(dH, len(H))
        L.bindTriInfo(dTI, len(mo.triInfo))
        for name, val, ty in (("k_numCubes", 50, np.uint32), ("k_totalNumCubes", 50 ** 3, np.uint32),
                              ("k_maxTrianglesPerCube", W, np.uint32), ("k_cubeLength", F(2.0) / F(50), F),
                              ("k_reflectionType", 1, np.uint32), ("k_permeability", case.permeability, F),
                              ("k_deltaTime", case.dt, F)):
            a = np.array([val], ty)
            L.copyConstantToDevice(name.encode(), a.ctypes.data, 0, 4)
        for name, tab in (("k_T2Values", case.T2), ("k_stdDevs", case.stdDevs)):
            a = np.ascontiguousarray(tab, F)
            L.copyConstantToDevice(name.encode(), a.ctypes.data, 0, 16)
        spins = np.zeros(case.N, np.dtype([("mag", "<f4"), ("phase", "<f4"), ("comp", "u1"), ("pad", "u1"),
                                           ("fiber", "<u2")]))
        spins["mag"], spins["phase"], spins["comp"], spins["fiber"] = case.mag, case.phase, case.comp, case.fiber
        dPos, dSeed, dSpins = dev(case.pos, 0), dev(np.zeros(2 * case.N, np.uint32), 0), dev(spins, 0)
        dD = [dev(d[k * its:(k + 1) * its].reshape(-1), 0) for k in range(2)]
        dCnt = dev(np.zeros(2 * case.N, np.uint32), 0)
        g = _lib.Float3(*[float(x) for x in case.g])
        for k in range(2):
            if k:
                mo, H, cc = meshes[1][:3]
                for dst, src in ((dV, mo.vertices), (dH, H), (dTI, mo.triInfo), (dTic, dense[1]), (dCc, cc)):
                    L.copyArrayToDevice(dst, src.ctypes.data, 0, src.nbytes)
            L.dsim3_set_replay(dD[k], dCnt)
            L.integrateSystem(dPos, dSeed, dSpins, float(case.dt), float(case.permeability), case.N, g, float(case.pc),
                              its, dTic, dCc)
            assert L.dsim3_last_status() == 0, L.dsim3_last_error()
        pos, out = np.zeros_like(case.pos), np.zeros_like(spins)
        L.copyArrayFromDevice(pos.ctypes.data, dPos, 0, pos.nbytes)
        L.copyArrayFromDevice(out.ctypes.data, dSpins, 0, out.nbytes)
    finally:
        L.dsim3_set_replay(None, None)
        L.unbindVertices(); L.unbindTriangleHelpers(); L.unbindTriInfo()
        for q in bases:
            L.freeArray(q)
    assert np.array_equal(pos.view(np.uint32), rpos.view(np.uint32))
    assert np.array_equal(out["mag"].view(np.uint32), mag.view(np.uint32))
    assert np.array_equal(out["comp"], comp.astype(np.uint8)) and np.array_equal(out["fiber"], fib.astype(np.uint16))
