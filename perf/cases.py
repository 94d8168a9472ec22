"""The work a user of this framework has it do, as measurable cases.

Each case is a dict of plain values; prepare() makes what a program holds before the call (substrate handles, spin
objects, initial spins, gradient tables), run() is one pass through the public entry points, exact() the same pass in
64 bits in plain torch.  Substrates are beaded tubes (dSim3 meshes) and packed cylinders (dSim2) in the shapes, step
lengths, waveforms and spin counts of the benchmark and of the job mixes (dsim_gb300/jobs.py)."""
import ctypes
import math

import numpy as np
import torch

from dsim_gb300 import _lib
from dsim_gb300 import engine as E
from dsim_gb300 import jobs as J
from dsim_gb300 import substrates as S

F = np.float32
GAMMA = 42576.0     # kHz/T
SCALE = 25.0        # um per normalised unit of the mesh box (50 um)
PITCH = 2.5         # um between tube centres
SPIN_RADIUS = 0.005


# ---- cases -----------------------------------------------------------------------------------------------------
def listed():
    return [
        # one updateSpins call of the sequencer (stepsPerUpdate = 20) and its signal: the smallest call there is
        dict(name="update_1k", kind="update", spins=1000, steps=20, tubes=9, verts=16, ring=1.0, membranes="G", perm=0.0),
        # one gradient on a few axons with myelin and exchange, few spins: a long chain of short steps
        dict(name="walk_mesh_4k", kind="walk", spins=4096, steps=600, tubes=25, verts=24, ring=0.5, membranes="AM",
             perm=0.01, find=False),
        # one gradient as the simulate call does it: fresh positions, compartments found on the GPU, walk, signal
        dict(name="walk_mesh_100k", kind="walk", spins=100001, steps=400, tubes=100, verts=32, ring=0.5,
             membranes="G", perm=0.0, find=True),
        # the headline workload's size: 2.56M triangles, 1M spins, 1000 steps
        dict(name="walk_mesh_1m", kind="walk", spins=1 << 20, steps=1000, tubes=400, verts=32, ring=0.5,
             membranes="G", perm=0.0, find=False),
        # the cylinder configuration: 64 Gamma-radius cylinders, 10,000 spins, dt 10 us, one gradient
        dict(name="walk_cyl_10k", kind="cyl", spins=10000, steps=1000, cylinders=64, perm=0.0, inner=0.7),
        # many spins on a larger packing with permeable membranes
        dict(name="walk_cyl_300k", kind="cyl", spins=300007, steps=400, cylinders=256, perm=0.005, inner=0.7),
        # a mix of mesh and cylinder jobs of different sizes in one batch, every gradient of every job
        dict(name="batch_mix", kind="batch", form="plain", jobs=6, lo=4096, hi=65536, steps=800, tubes=100, verts=32,
             ring=0.5, cylinders=64, dirs=32, perm=0.0),
        # the same in the forms that hold the signal error bar: cell-local, permeable
        dict(name="batch_local", kind="batch", form="local", jobs=4, lo=4096, hi=65536, steps=500, tubes=100, verts=32,
             ring=0.5, cylinders=64, dirs=32, perm=0.002),
        # and in FP64
        dict(name="batch_fp64", kind="batch", form="precise", jobs=2, lo=8192, hi=16384, steps=300, tubes=25, verts=32,
             ring=0.5, cylinders=64, dirs=16, perm=0.0),
        # a gradient table read from one walk's moments: 128 directions x 3 b-values (free water, a control run)
        dict(name="readout_384", kind="readout", spins=65537, steps=64, cylinders=64, dirs=128),
        # the reference's plugin call on device arrays the caller owns
        dict(name="plugin_64k", kind="plugin", spins=65536, steps=100, tubes=100, verts=32, ring=0.5, membranes="G",
             perm=0.0),
        # reading a substrate in: records, reference grid, fine grid
        dict(name="build_640k", kind="build", tubes=100, verts=32, ring=0.5, membranes="G"),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["update", "walk", "walk", "walk", "cyl", "cyl", "batch", "batch", "readout", "plugin", "build"])
    mesh = dict(tubes=rng.choice([9, 25, 49, 100, 196, 400]), verts=rng.choice([12, 16, 24, 32]),
                ring=rng.choice([0.5, 0.8, 1.0]))
    perm = rng.choice([0.0, 0.0, float("%.3g" % math.exp(rng.uniform(math.log(1e-4), math.log(1e-2))))])
    if kind == "update":
        return dict(kind=kind, spins=log(500, 5000), steps=rng.randint(1, 50), tubes=rng.choice([9, 16]),
                    verts=rng.choice([12, 16]), ring=1.0, membranes=rng.choice(["G", "AM"]), perm=perm)
    if kind == "walk":
        n = log(1000, 1 << 20)
        return dict(kind=kind, spins=n, steps=max(50, min(log(100, 1000), int(4e8 / n))), membranes=rng.choice(["G", "AM"]),
                    perm=perm, find=rng.random() < 0.5, **mesh)
    if kind == "cyl":
        n = log(1000, 1 << 20)
        return dict(kind=kind, spins=n, steps=max(50, min(log(100, 2000), int(4e8 / n))),
                    cylinders=rng.choice([16, 64, 144, 256]), perm=perm, inner=rng.choice([0.6, 0.7, 0.8]))
    if kind == "batch":
        form = rng.choice(["plain", "plain", "local", "precise"])
        top = {"plain": 65536, "local": 32768, "precise": 8192}[form]
        return dict(kind=kind, form=form, jobs=rng.randint(1, 6), lo=1000, hi=top, steps=log(100, 600),
                    tubes=mesh["tubes"], verts=mesh["verts"], ring=mesh["ring"], cylinders=64, dirs=rng.randint(6, 64), perm=perm)
    if kind == "readout":
        return dict(kind=kind, spins=log(4096, 150000), steps=rng.randint(16, 100), cylinders=64, dirs=rng.randint(6, 128))
    if kind == "plugin":
        return dict(kind=kind, spins=log(1000, 200000), steps=rng.randint(10, 300), membranes="G", perm=perm,
                    tubes=rng.choice([9, 25, 100]), verts=mesh["verts"], ring=mesh["ring"])
    return dict(kind=kind, membranes=rng.choice(["G", "AM"]), **mesh)


# ---- substrates (the same for every seed: a program reads them once) ---------------------------------------------
_made = {}


def _once(key, make):
    if key not in _made:
        _made[key] = make()
    return _made[key]


def _tubes(c):
    """Beaded tubes along z on a jittered square lattice in the 50 um box: radii log-normal, clipped so that no two
    tubes touch (myelin, where there is one, at 1.25 r); as substrates.beaded_tubes lays its arrays out."""
    membranes = c.get("membranes", "G")
    key = ("tubes", c["tubes"], c["verts"], c["ring"], membranes)

    def make():
        rng = np.random.default_rng(17 * c["tubes"] + c["verts"])
        k = int(math.isqrt(c["tubes"]))
        layers = [(2, 1.0)] if membranes == "G" else [(0, 1.0), (1, 1.25)]
        fit = PITCH / 2 / 1.2 / layers[-1][1] - 0.02
        r0 = np.clip(rng.lognormal(0.0, 0.4, k * k), 0.4, fit)
        ij = np.stack(np.meshgrid(np.arange(k), np.arange(k), indexing="ij"), -1).reshape(-1, 2)
        room = PITCH / 2 - 0.01 - 1.2 * layers[-1][1] * r0
        xy = (ij - (k - 1) / 2.0) * PITCH + rng.uniform(-1, 1, (k * k, 2)) * room[:, None]
        V, T, mem, fib, nv = [], [], [], [], 0
        for i in range(k * k):
            for kind, grow in layers:
                v, t = S.tube_mesh(xy[i, 0], xy[i, 1], lambda z: grow * r0[i] * (1 + 0.2 * np.sin(2 * np.pi * z / 10.0)),
                                   -25.0, 25.0, c["ring"], c["verts"], v_offset=nv)
                V.append(v), T.append(t)
                mem.append(np.full(len(t), kind, np.uint32)), fib.append(np.full(len(t), i, np.uint32))
                nv += len(v)
        return dict(vertices=np.concatenate(V).astype(F), trgls=np.concatenate(T).astype(np.uint32),
                    membrane=np.concatenate(mem), fiber=np.concatenate(fib), centres=xy, radii=r0, k=k, layers=layers)

    return _once(key, make)


def _mesh(c):
    t = _tubes(c)
    key = ("mesh", c["tubes"], c["verts"], c["ring"], c.get("membranes", "G"))
    return _once(key, lambda: E.Mesh.from_arrays(t["vertices"], t["trgls"], t["membrane"], t["fiber"], SCALE))


def _start_mesh(c, n, rng):
    """Uniform positions over the tubes' square, and each spin's compartment and fiber from the geometry."""
    t = _tubes(c)
    half = t["k"] * PITCH / 2.0 / SCALE
    pos = np.empty((n, 3), F)
    pos[:, :2] = rng.random((n, 2), F) * F(1.98 * half) - F(0.99 * half)
    pos[:, 2] = rng.random(n, F) * F(1.98) - F(0.99)
    um = pos.astype(np.float64) * SCALE
    ij = np.clip(np.floor(um[:, :2] / PITCH + t["k"] / 2.0).astype(np.int64), 0, t["k"] - 1)
    fib = ij[:, 0] * t["k"] + ij[:, 1]
    d = np.hypot(um[:, 0] - t["centres"][fib, 0], um[:, 1] - t["centres"][fib, 1])
    r = t["radii"][fib] * (1 + 0.2 * np.sin(2 * np.pi * um[:, 2] / 10.0))
    facet = math.cos(math.pi / c["verts"])
    comp = np.zeros(n, np.uint8)
    if c.get("membranes", "G") == "G":
        comp[d < r * facet] = 3
    else:
        comp[d < 1.25 * r * facet] = 2
        comp[d < r * facet] = 1
    return pos, comp, np.where(comp > 0, fib, 0xFFFF).astype(np.uint16)


def _packing(n):
    """n cylinders at half the area of a square cell (numpy's own relaxation, from the package's generator)."""
    cell = 20.0 * math.sqrt(n / 64.0)
    return _once(("xy", n), lambda: S.packed_cylinders(n=n, cell=cell, fraction=0.5, seed=3)) + (cell / 2.0,)


def _cylinders(n):
    xy, r, ss = _packing(n)
    return _once(("cyl", n), lambda: E.Cylinders.from_arrays(*S.cylinders_normalised(xy, r, ss)))


def _start_cyl(n_cyl, n, rng, inner):
    xy, r, ss = _packing(n_cyl)
    pos = rng.random((n, 3), F) * F(1.98) - F(0.99)
    p = torch.from_numpy(pos).cuda().double()[:, :2] * ss
    d = torch.hypot(p[:, None, 0] - torch.as_tensor(xy[:, 0]).cuda(), p[:, None, 1] - torch.as_tensor(xy[:, 1]).cuda())
    d, near = (d / torch.as_tensor(r).cuda()).min(1)
    d, near = d.cpu().numpy(), near.cpu().numpy()
    imo = np.where(d < inner, 0, np.where(d <= 1.0, 1, 2)).astype(np.uint32)
    return pos, imo, np.where(imo < 2, near, 0xFFFFFFFF).astype(np.uint32)


# ---- waveforms and parameters ------------------------------------------------------------------------------------
def _pgse(steps):
    """+1 over the first 0.3 of the walk, -1 over 0.3 from 0.6 on."""
    w = np.zeros(steps, F)
    a, b = max(1, round(0.3 * steps)), round(0.6 * steps)
    w[:a] = 1
    w[b:b + a] = -1
    return w


def _strength(steps, dt, b=2.0):
    T = steps * dt
    return min(300.0, J.pgse_gmag(b, 0.3 * T, 0.6 * T))


MESH_DT, MESH_D, MESH_T2 = 0.005, 2.0, (80.0, 70.0, 7.5, 80.0)
CYL_DT, CYL_ADC, CYL_T2 = 0.01, (2.0, 2.0, 0.2), (70.0, 8.0, 80.0)  # intra, extra, myelin; fiber, myelin, outside
DIRECTION = np.array([0.8, 0.36, 0.48])


def _gradient(steps, dt, scale):
    g = E.grad_scaled(_strength(steps, dt) * DIRECTION, scale).astype(F)
    return (_pgse(steps)[:, None] * g[None, :]).astype(F)


def _job_sizes(c, rng):
    out = []
    for k in range(c["jobs"]):
        n = int(round(math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"])))))
        out.append((k % 2 == 1, n, int(c["steps"] * rng.uniform(0.5, 1.0)), float(rng.uniform(0.005, 0.010))))
    return out


# ---- prepare and run ---------------------------------------------------------------------------------------------
def prepare(c, seed):
    rng = np.random.default_rng(seed)
    s = dict(c=c, seed=int(seed))
    kind = c["kind"]
    if kind in ("update", "walk"):
        n = c["spins"]
        s["mesh"], s["spins"] = _mesh(c), E.Spins(n)
        s["pos"], s["comp"], s["fiber"] = _start_mesh(c, n, rng)
        s["one"], s["zero"] = np.ones(n, F), np.zeros(n, F)
        s["params"] = E.mesh_params(E.std_devs(MESH_D, MESH_D, 0.1 * MESH_D, SCALE, MESH_DT), MESH_T2, c["perm"], MESH_DT,
                                    E.phase_constant(GAMMA, MESH_DT))
        s["grad"] = _gradient(c["steps"], MESH_DT, SCALE)
        if kind == "update":
            s["spins"].set(s["pos"], s["one"], s["zero"], s["comp"], s["fiber"])
            s["g"] = E.grad_scaled(80.0 * DIRECTION, SCALE).astype(F)
            s["step"] = 0
    elif kind == "cyl":
        n = c["spins"]
        ss = _packing(c["cylinders"])[2]
        s["cyl"], s["spins"] = _cylinders(c["cylinders"]), E.Spins(n)
        s["pos"], s["imo"], s["near"] = _start_cyl(c["cylinders"], n, rng, c["inner"])
        s["params"] = E.cyl_params(*CYL_ADC, ss, *CYL_T2, c["perm"], c["inner"], CYL_DT, E.phase_constant(GAMMA, CYL_DT))
        s["grad"] = _gradient(c["steps"], CYL_DT, ss)
    elif kind == "batch":
        s["jobs"] = []
        sizes = _job_sizes(c, np.random.default_rng(c["jobs"] * 1000 + c["steps"]))  # the mix is the case's, not the seed's
        s["batch"] = E.Batch(sum((n + 31) // 32 * 32 for _, n, _, _ in sizes), len(sizes))
        sub = (s["batch"].add_mesh(_mesh(c)), s["batch"].add_cyl(_cylinders(c["cylinders"])))
        for k, (cyl, n, steps, dt) in enumerate(sizes):
            T = steps * dt
            common = dict(steps=steps, dt=F(dt), phase_constant=E.phase_constant(GAMMA, dt), seed=seed * 100 + k,
                          permeability=c["perm"], delta=0.3 * T, Delta=0.6 * T, precise=c["form"] == "precise",
                          local=c["form"] == "local")
            if cyl:
                ss = _packing(c["cylinders"])[2]
                pos, comp, fib = _start_cyl(c["cylinders"], n, rng, 0.7)
                sd = [math.sqrt(2 * a / ss ** 2 * dt) for a in (CYL_ADC[0], CYL_ADC[2], CYL_ADC[1])]
                common.update(step_sd=sd, T2=CYL_T2, inner_radius_proportion=0.7)
            else:
                ss = SCALE
                pos, comp, fib = _start_mesh(c, n, rng)
                common.update(step_sd=E.std_devs(MESH_D, MESH_D, 0.1 * MESH_D, ss, dt), T2=MESH_T2)
            dirs = J.fibonacci_dirs(c["dirs"])
            G = np.concatenate([min(300.0, J.pgse_gmag(b, 0.3 * T, 0.6 * T)) * dirs for b in (1.0, 2.0, 3.0)])
            s["jobs"].append((sub[cyl], n, pos, comp.astype(np.uint8), fib.astype(np.uint32), common, E.grad_scaled(G, ss)))
    elif kind == "readout":
        n, steps = c["spins"], c["steps"]
        ss = _packing(c["cylinders"])[2]
        pos, imo, near = _start_cyl(c["cylinders"], n, rng, 0.7)
        s["batch"] = E.Batch((n + 31) // 32 * 32, 1)
        sub = s["batch"].add_cyl(_cylinders(c["cylinders"]))
        sd = [math.sqrt(2 * a / ss ** 2 * CYL_DT) for a in (CYL_ADC[0], CYL_ADC[2], CYL_ADC[1])]
        s["job"] = s["batch"].submit(sub, pos, imo.astype(np.uint8), near, steps, CYL_DT, sd, CYL_T2,
                                     E.phase_constant(GAMMA, CYL_DT), seed, permeability=1.0, waveform="table",
                                     table=_pgse(steps), inner_radius_proportion=0.7)
        s["batch"].run()
        s["G"] = _table(c, ss)
    elif kind == "plugin":
        _prepare_plugin(s, c, rng)
    elif kind == "build":
        t = _tubes(c)  # its triangles and vertices with another tube first
        k, each = int(rng.integers(c["tubes"])), {n: len(t[n]) // c["tubes"] for n in ("vertices", "trgls")}
        at = np.roll(t["trgls"], k * each["trgls"], axis=0).astype(np.int64) + k * each["vertices"]
        s["arrays"] = dict(t, vertices=np.roll(t["vertices"], k * each["vertices"], axis=0),
                           trgls=(at % len(t["vertices"])).astype(np.uint32))
    return s


def _table(c, ss):
    dirs = J.fibonacci_dirs(c["dirs"])
    return E.grad_scaled(np.concatenate([f * _strength(c["steps"], CYL_DT, 3.0) * dirs for f in (0.58, 0.82, 1.0)]), ss)


def _prepare_plugin(s, c, rng):
    """The arrays the reference's host code allocates, binds and passes, as device tensors of the caller's."""
    mesh, n = _mesh(c), c["spins"]

    def arrays():
        v, ti = mesh.arrays()
        start, tri = mesh.grid()
        tri3 = _tubes(c)["trgls"].astype(np.int64)
        p = v.reshape(-1, 3)[tri3]
        a, b = p[:, 2] - p[:, 0], p[:, 1] - p[:, 0]
        nrm = np.cross(a, b)
        nrm = nrm / np.sqrt((nrm * nrm).sum(1, dtype=F))[:, None]
        # triangleHelpers: normal, u, v, uv, uu, vv
        h = np.concatenate([nrm, a, b, (a * b).sum(1)[:, None], (a * a).sum(1)[:, None], (b * b).sum(1)[:, None]], 1)
        cnt = np.diff(start.astype(np.int64))
        dense = np.zeros((len(cnt), int(cnt.max())), np.uint32)
        at = np.arange(len(tri)) - np.repeat(start[:-1].astype(np.int64), cnt)
        dense[np.repeat(np.arange(len(cnt)), cnt), at] = tri
        dev = [torch.from_numpy(np.ascontiguousarray(x).view(np.int32).reshape(-1)).cuda()
               for x in (v, h.astype(F), ti, dense, cnt.astype(np.uint32))]
        return dev, dense.shape[1]

    key = ("plugin", c["tubes"], c["verts"], c["ring"])
    s["bound"], most = _once(key, arrays)
    L = s["lib"] = _lib.abi3()
    V, H, TI, tic, cc = s["bound"]
    L.bindVertices(V.data_ptr(), V.numel())
    L.bindTriangleHelpers(H.data_ptr(), H.numel())
    L.bindTriInfo(TI.data_ptr(), TI.numel())
    sd = E.std_devs(MESH_D, MESH_D, 0.1 * MESH_D, SCALE, MESH_DT)
    tables = [(b"k_stdDevs", np.array(sd, F)), (b"k_T2Values", np.array(MESH_T2, F))]
    plain = [(b"k_numCubes", np.uint32(50)), (b"k_totalNumCubes", np.uint32(50 ** 3)),
             (b"k_maxTrianglesPerCube", np.uint32(most)), (b"k_cubeLength", F(2.0) / F(50)), (b"k_reflectionType", np.uint32(1)),
             (b"k_deltaTime", F(MESH_DT)), (b"k_permeability", F(c["perm"]))]
    for name, v in tables + [(k, np.array([x])) for k, x in plain]:
        L.copyConstantToDevice(name, v.ctypes.data, 0, v.nbytes)
    pos, comp, fib = _start_mesh(c, n, rng)
    rec = np.zeros(n, dtype=[("m", F), ("p", F), ("c", np.uint8), ("x", np.uint8), ("f", np.uint16)])
    rec["m"], rec["c"], rec["f"] = 1.0, comp, fib
    s["pos"] = torch.from_numpy(pos.reshape(-1)).cuda()
    s["keys"] = torch.from_numpy(rng.integers(1, 1 << 31, 2 * n).astype(np.int32)).cuda()
    s["rec"] = torch.from_numpy(rec.view(np.uint8).reshape(n, 12)).cuda()
    s["g"] = E.grad_scaled(80.0 * DIRECTION, SCALE).astype(F)


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "update":
        sp = s["spins"]
        E.mesh_run(s["mesh"], sp, s["params"], s["g"], c["steps"], seed=s["seed"], step0=s["step"])
        s["step"] += c["steps"]
        return [sp.signal(), *sp.get()]
    if kind == "walk":
        sp = s["spins"]
        sp.set(s["pos"], s["one"], s["zero"], s["comp"], s["fiber"])
        if c["find"]:
            s["mesh"].compartments(sp, seed=s["seed"])
        E.mesh_run(s["mesh"], sp, s["params"], iterations=c["steps"], seed=s["seed"], grad_per_step=s["grad"])
        return [sp.signal(), *sp.get()]
    if kind == "cyl":
        sp = s["spins"]
        sp.set_cyl(s["pos"], None, None, s["imo"], s["near"])
        E.cyl_run(s["cyl"], sp, s["params"], iterations=c["steps"], seed=s["seed"], grad_per_step=s["grad"])
        return [sp.signal(0.8), *sp.get_cyl()]
    if kind == "batch":
        b = s["batch"]
        ids = [b.submit(sub, pos, comp, fib, **kw) for sub, n, pos, comp, fib, kw, G in s["jobs"]]
        b.run()
        out = []
        for jid, (sub, n, pos, comp, fib, kw, G) in zip(ids, s["jobs"]):
            out.append([b.signal(jid, G), *b.get(jid, n)])
        for jid in ids:
            b.retire(jid)
        b.compact()
        return out
    if kind == "readout":
        return s["batch"].signal(s["job"], s["G"])
    if kind == "plugin":
        L, (V, H, TI, tic, cc) = s["lib"], s["bound"]
        L.integrateSystem(s["pos"].data_ptr(), s["keys"].data_ptr(), s["rec"].data_ptr(), MESH_DT, c["perm"], c["spins"],
                          _lib.Float3(*[float(x) for x in s["g"]]), float(E.phase_constant(GAMMA, MESH_DT)), c["steps"],
                          tic.data_ptr(), cc.data_ptr())
        return [s["pos"], s["keys"], s["rec"]]
    a = s["arrays"]
    m = E.Mesh.from_arrays(a["vertices"], a["trgls"], a["membrane"], a["fiber"], SCALE)
    out = [*(x.view(np.int32) for x in m.grid()), m.nonempty, m.max_per_cell]
    m.free()
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------------
def work(c):
    """Bytes: the substrate's records and each spin's state read once, the state (and the signal) written once.
    Operations of a spin-step: ten Philox rounds, Box-Muller, the move, one membrane test, decay and phase."""
    kind = c["kind"]
    tri = 2 * c["tubes"] * c["verts"] * round(50 / c["ring"]) * (2 if c.get("membranes") == "AM" else 1) if "tubes" in c else 0
    mesh_step, cyl_step = 250.0, 200.0
    if kind in ("update", "walk"):
        return dict(bytes=64.0 * tri + 2 * 23.0 * c["spins"], flops=mesh_step * c["spins"] * c["steps"])
    if kind == "cyl":
        return dict(bytes=2 * 28.0 * c["spins"], flops=cyl_step * c["spins"] * c["steps"])
    if kind == "batch":
        by, fl = 64.0 * tri, 0.0
        for cyl, n, steps, _ in _job_sizes(c, np.random.default_rng(c["jobs"] * 1000 + c["steps"])):
            by += (17.0 + 45.0) * n + 3 * c["dirs"] * 120
            fl += n * steps * (cyl_step if cyl else mesh_step) + n * 3 * c["dirs"] * 60.0
        return dict(bytes=by, flops=fl)
    if kind == "readout":
        return dict(bytes=28.0 * c["spins"] + 360.0 * c["dirs"], flops=60.0 * 3 * c["dirs"] * c["spins"])
    if kind == "plugin":
        return dict(bytes=100.0 * tri + 2 * 32.0 * c["spins"], flops=mesh_step * c["spins"] * c["steps"])
    return dict(bytes=20.0 * tri + 6.0 * tri + 64.0 * tri, flops=100.0 * tri)


# ---- the same in 64 bits -----------------------------------------------------------------------------------------
def _philox(spin, step, k0, k1):
    """Four 32-bit words per spin of Philox4x32-10 (Salmon et al., SC'11), counter (spin, step, 0, 0)."""
    m = 0xFFFFFFFF

    def mul(a, x):
        hi = (a * (x >> 16) + ((a * (x & 0xFFFF)) >> 16)) >> 16
        return hi, (a * x) & m

    a, b, c, d = spin, torch.full_like(spin, step), torch.zeros_like(spin), torch.zeros_like(spin)
    for r in range(10):
        h0, l0 = mul(0xD2511F53, a)
        h1, l1 = mul(0xCD9E8D57, c)
        a, b, c, d = h1 ^ b ^ ((k0 + r * 0x9E3779B9) & m), l1, h0 ^ d ^ ((k1 + r * 0xBB67AE85) & m), l0
    return a, b, c, d


def _steps64(spin, step, seed):
    """Three normals and the uniform of one step (Box-Muller on the four words)."""
    a, b, c, d = _philox(spin, step, seed & 0xFFFFFFFF, seed >> 32)
    r1 = torch.sqrt(-2 * torch.log((a.double() + 0.5) / 2 ** 32))
    r2 = torch.sqrt(-2 * torch.log((c.double() + 0.5) / 2 ** 32))
    t1 = (b >> 8).double() / 2 ** 24 * 2 * math.pi
    u = ((d >> 8) + 1).double() / 2 ** 24
    return torch.stack([r1 * torch.cos(t1), r1 * torch.sin(t1), r2 * torch.cos(u * 2 * math.pi)], 1), u


def _sums64(mag, phase, comp, keep=None):
    out = torch.zeros(5, 3, dtype=torch.float64)
    for k in range(5):
        on = torch.ones_like(mag, dtype=torch.bool) if k == 0 else comp == k - 1
        on = on if keep is None else on & keep
        out[k] = torch.stack([(mag * torch.cos(phase))[on].sum(), (mag * torch.sin(phase))[on].sum(), on.sum().double()]).cpu()
    return out


def exact(c, seed):
    """Mesh walks that plain tensors can follow, and the readout.  A walk among cylinders has no value here: dSim2's
    cell lists, which decide the membranes a step meets, leave out a few per cent of the fibers near cell borders."""
    kind = c["kind"]
    with torch.no_grad():
        if kind == "readout":
            return _exact_readout(c, seed)
        if kind == "update" or (kind == "walk" and not c["find"] and c["spins"] * c["steps"] <= 4e6):
            return _exact_mesh(c, seed)
    return None


def _clamp(p):
    return p.clamp(-1 + SPIN_RADIUS, 1 - SPIN_RADIUS)


def _exact_readout(c, seed):
    """A free walk's moments and every gradient's phases."""
    ss = _packing(c["cylinders"])[2]
    pos, imo, _ = _start_cyl(c["cylinders"], c["spins"], np.random.default_rng(seed), 0.7)
    x = torch.from_numpy(pos).cuda().double()
    imo = torch.from_numpy(imo.astype(np.int64)).cuda()
    sd = torch.tensor([math.sqrt(2 * a / ss ** 2 * CYL_DT) for a in (CYL_ADC[0], CYL_ADC[2], CYL_ADC[1])]).cuda().double()
    decay = (1 - CYL_DT / torch.tensor(CYL_T2).cuda().double()[imo]) ** c["steps"]
    M, w, spin = torch.zeros_like(x), _pgse(c["steps"]), torch.arange(len(x), device="cuda")
    for it in range(c["steps"]):
        z, _u = _steps64(spin, it, seed)
        x = _clamp(x + z * sd[imo][:, None])
        M += float(w[it]) * x
    G = torch.from_numpy(np.ascontiguousarray(_table(c, ss))).cuda().double() * (2 * math.pi * GAMMA * CYL_DT)
    return torch.stack([_sums64(decay, M @ g, imo) for g in G])


def _exact_mesh(c, seed):
    """dSim3's step: the nearest triangle on the way reflects the rest of the step or lets the spin through."""
    t = _tubes(c)
    pos, comp, fib = _start_mesh(c, c["spins"], np.random.default_rng(seed))
    x = torch.from_numpy(pos).cuda().double()
    comp, fib = torch.from_numpy(comp.astype(np.int64)).cuda(), torch.from_numpy(fib.astype(np.int64)).cuda()
    V = torch.from_numpy(t["vertices"] / F(SCALE)).cuda().double()
    tri = V[torch.from_numpy(t["trgls"].astype(np.int64)).cuda()]
    p0, e1, e2 = tri[:, 0], tri[:, 2] - tri[:, 0], tri[:, 1] - tri[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    uu, uv, vv = (e1 * e1).sum(1), (e1 * e2).sum(1), (e2 * e2).sum(1)
    D = uv * uv - uu * vv
    mem = torch.from_numpy(t["membrane"].astype(np.int64)).cuda()
    of = torch.from_numpy(t["fiber"].astype(np.int64)).cuda()
    table, n = _buckets(tri)
    sd = torch.from_numpy(np.array(E.std_devs(MESH_D, MESH_D, 0.1 * MESH_D, SCALE, MESH_DT))).cuda().double()
    T2 = torch.tensor(MESH_T2).cuda().double()
    if c["kind"] == "walk":
        grad = torch.from_numpy(_gradient(c["steps"], MESH_DT, SCALE)).cuda().double()
    else:
        grad = torch.from_numpy(E.grad_scaled(80.0 * DIRECTION, SCALE).astype(F)).cuda().double().expand(c["steps"], 3)
    pc, perm = 2 * math.pi * GAMMA * MESH_DT, c["perm"]
    N = len(x)
    spin = torch.arange(N, device="cuda")
    mag, ph = torch.ones(N, device="cuda").double(), torch.zeros(N, device="cuda").double()
    for it in range(c["steps"]):
        z, u = _steps64(spin, it, seed)
        p = x + z * sd[comp][:, None]
        o, live = x.clone(), spin
        last = torch.full_like(spin, -1)
        umax, umin = torch.ones_like(u), torch.zeros_like(u)
        for _ in range(64):
            hit, at = _first_hit(table, n, p0, e1, e2, nrm, uu, uv, vv, D, o[live], p[live], last[live])
            on = hit >= 0
            live, hit, at = live[on], hit[on], at[on]
            if len(live) == 0:
                break
            thr = umax[live] - (umax[live] - umin[live]) * perm
            off = u[live] <= thr
            a, h = live[off], hit[off]
            s = p[a] - at[off]
            p[a] = at[off] + s - 2 * nrm[h] * (nrm[h] * s).sum(1, keepdim=True)
            umax[a] = thr[off]
            a, h = live[~off], hit[~off]
            umin[a] = thr[~off]
            was, m = comp[a], mem[h]
            to = torch.where(was == 2, torch.where(m == 0, 1, 0), torch.where(was == 1, 2, torch.where(was == 3, 0, torch.where(m == 1, 2, 3))))
            fib[a] = torch.where(was == 0, of[h], torch.where(to == 0, 0xFFFF, fib[a]))
            comp[a] = to
            o[live], last[live] = at, hit
        x = _clamp(p)
        mag = mag - mag / T2[comp] * MESH_DT
        ph = ph + (x * grad[it]).sum(1) * pc
    return [_sums64(mag, ph, comp), x.reshape(-1).cpu(), mag.cpu(), ph.cpu(), None, None]


def _buckets(tri, n=50):
    """A padded list of the triangles whose bounding box meets each cell of an n^3 grid."""
    lo = ((tri.amin(1) + 1) * n / 2 - 1e-4).floor().clamp(0, n - 1).long()
    hi = ((tri.amax(1) + 1) * n / 2 + 1e-4).floor().clamp(0, n - 1).long()
    w = hi - lo + 1
    cnt = w.prod(1)
    who = torch.repeat_interleave(torch.arange(len(tri), device="cuda"), cnt)
    at = torch.arange(len(who), device="cuda") - (cnt.cumsum(0) - cnt)[who]
    cell = lo[who] + torch.stack([at // (w[who, 1] * w[who, 2]), at // w[who, 2] % w[who, 1], at % w[who, 2]], 1)
    cell = (cell[:, 0] * n + cell[:, 1]) * n + cell[:, 2]
    order = cell.argsort(stable=True)
    cell, who = cell[order], who[order]
    per = torch.bincount(cell, minlength=n ** 3)
    table = torch.full((n ** 3, int(per.max())), -1, device="cuda", dtype=torch.long)
    table[cell, torch.arange(len(cell), device="cuda") - (per.cumsum(0) - per)[cell]] = who
    return table, n


def _first_hit(table, n, p0, e1, e2, nrm, uu, uv, vv, D, o, p, last, most=4096):
    hits, ats = [], []
    for k in range(0, len(o), most):
        a, b, ex = o[k:k + most], p[k:k + most], last[k:k + most]
        lo = ((torch.minimum(a, b) + 1) * n / 2).floor().clamp(0, n - 1).long()
        hi = ((torch.maximum(a, b) + 1) * n / 2).floor().clamp(0, n - 1).long()
        wx, wy, wz = (int(v) + 1 for v in (hi - lo).amax(0))
        step = torch.cartesian_prod(*(torch.arange(v, device="cuda") for v in (wx, wy, wz))).reshape(-1, 3)
        cell = torch.minimum(lo[:, None] + step, hi[:, None])
        cand = table[(cell[..., 0] * n + cell[..., 1]) * n + cell[..., 2]].reshape(len(a), -1)
        q = cand.clamp(min=0)
        d = (b - a)[:, None]
        den = (nrm[q] * d).sum(2)
        r = (nrm[q] * (p0[q] - a[:, None])).sum(2) / den
        w = a[:, None] + r[..., None] * d - p0[q]
        wu, wv = (w * e1[q]).sum(2), (w * e2[q]).sum(2)
        s, tt = (uv[q] * wv - vv[q] * wu) / D[q], (uv[q] * wu - uu[q] * wv) / D[q]
        ok = (cand >= 0) & (cand != ex[:, None]) & (r > 0) & (r < 1) & (s >= 0) & (tt >= 0) & (s + tt <= 1)
        r = torch.where(ok, r, torch.full_like(r, 2.0))
        best, j = r.min(1)
        hits.append(torch.where(best < 1.5, q.gather(1, j[:, None])[:, 0], -1))
        ats.append(a + best[:, None] * (b - a))
    if not hits:
        return torch.zeros(0, device="cuda", dtype=torch.long), o
    return torch.cat(hits), torch.cat(ats)
