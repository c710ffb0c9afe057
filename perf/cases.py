"""The performance cases of this framework: what a user's program has it do, over the range of sizes.

Almost all the work of a shallow-water run is the implicit time step (:meth:`SW2GPU.step`), called
as the reference's time loop calls ``fe_sw2_solve``: the caller holds the state on the host, hands
over the two time levels the step reads and takes the new one back.  The cases are that call from
the 2,000-node channel to the million-triangle basin, in plain FP64 and on the mixed path, with the
CUDA-graph option of small meshes, with the exact banded solve that the reference's default deck
setting (OP BLK 1) selects, with constituents carried along, and as an ensemble in the
continuous-batching engine; and the linear solve in the caller's own device memory.
"""
import ctypes
import dataclasses
import functools
import math

import numpy as np
import torch

from adhv8_kraken_b200 import capi, meshgen
from adhv8_kraken_b200.model import Constituent
from adhv8_kraken_b200.sw2 import SW2GPU, SW2Engine, lib

PRECISION = {"fp64": capi.SW2GPU_FP64, "mixed": capi.SW2GPU_MIXED}


def listed():
    return [
        # the rectangular channel of the tests and the benchmark: 4,000 triangles, the smallest call
        # a program makes in earnest, where launches and grid barriers are the time
        dict(name="channel_4k", kind="step", mesh="channel", nx=100, ny=20, precision="fp64", steps=1, graphs=0, solver="bjacobi"),
        # the same mesh as a resident run of four steps, each one graph launch
        dict(name="channel_4k_graph", kind="step", mesh="channel", nx=100, ny=20, precision="fp64", steps=4, graphs=2, solver="bjacobi"),
        # a mesh of the size of the reference's own test decks, whose OP BLK 1 asks for the exact solve
        dict(name="channel_2k_exact", kind="step", mesh="channel", nx=100, ny=10, precision="fp64", steps=1, graphs=0, solver="band"),
        # a small wet/dry basin with an odd node count
        dict(name="basin_7k", kind="step", mesh="basin", points=3517, precision="fp64", steps=2, graphs=0, solver="bjacobi"),
        # a median member of the ensemble on the mixed path
        dict(name="basin_32k_mixed", kind="step", mesh="basin", points=16001, precision="mixed", steps=1, graphs=0, solver="bjacobi"),
        # the ensemble's largest members, and an ordinary regional mesh
        dict(name="basin_200k", kind="step", mesh="basin", points=100000, precision="fp64", steps=1, graphs=0, solver="bjacobi"),
        dict(name="basin_260k_mixed", kind="step", mesh="basin", points=130007, precision="mixed", steps=1, graphs=0, solver="bjacobi"),
        # the benchmark's basin
        dict(name="basin_1M", kind="step", mesh="basin", points=500000, precision="fp64", steps=1, graphs=0, solver="bjacobi"),
        # flow and one constituent, on the channel and on a regional basin, with the mass balance kept
        dict(name="transport_4k", kind="transport", mesh="channel", nx=100, ny=20, constituents=1),
        dict(name="transport_150k", kind="transport", mesh="basin", points=75001, constituents=2),
        # an ensemble of uneven basins stepped together
        dict(name="engine_12", kind="engine", members=12, lo=5000, hi=40000, precision="fp64", steps=2),
        # a coupled model's linear solve in its own device memory, near the documented size limit
        dict(name="solve_14k_nodes", kind="solve", mesh="channel", nx=232, ny=59),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["transport"] * 2 + ["engine", "solve"])
    if kind == "engine":
        return dict(kind=kind, members=rng.randint(3, 12), lo=5000, hi=rng.randint(8000, 40000), precision="fp64",
                    steps=rng.randint(1, 2))
    if kind == "solve":
        return dict(kind=kind, mesh="channel", nx=rng.randint(50, 265), ny=rng.randint(9, 60))
    if kind == "transport":
        if rng.random() < 0.4:
            return dict(kind=kind, mesh="channel", nx=rng.randint(30, 200), ny=rng.randint(7, 40), constituents=rng.randint(1, 2))
        return dict(kind=kind, mesh="basin", points=_log(rng, 1000, 120000), constituents=rng.randint(1, 2))
    what = rng.choice(["channel", "basin", "basin", "basin", "exact"])
    if what == "exact":
        return dict(kind=kind, mesh="channel", nx=rng.randint(40, 120), ny=rng.randint(5, 16), precision="fp64", steps=1, graphs=0,
                    solver="band")
    if what == "channel":
        return dict(kind=kind, mesh="channel", nx=rng.randint(50, 300), ny=rng.randint(9, 60),
                    precision=rng.choice(["fp64", "mixed"]), steps=rng.randint(1, 4), graphs=rng.choice([0, 1, 2]), solver="bjacobi")
    precision = rng.choice(["fp64", "mixed"])
    points = _log(rng, 1000, 400000 if precision == "fp64" else 150000)
    return dict(kind=kind, mesh="basin", points=points, precision=precision,
                steps=rng.randint(1, 3) if points < 30000 else 1, graphs=rng.choice([0, 0, 2]) if points < 30000 else 0, solver="bjacobi")


# A program builds its mesh once and runs many states on it: the meshes of the last cases are kept.
@functools.lru_cache(maxsize=64)
def _basin(points, seed=2024, dt=5.0):
    """The benchmark's wet/dry basin at its resolution, whatever the size: a sloping bed with bumps
    whose tops are dry, 32 roughness classes, an inflow ramp in the west, a tailwater in the east.
    The nodes are those of a mesh generator, not of random points: a jittered grid without slivers,
    each quadrilateral cut along its Delaunay diagonal, in Morton order."""
    m = meshgen.bumpy_basin(600, seed, dt=dt)   # strings, materials, series and parameters
    rng = np.random.Generator(np.random.PCG64([seed, points]))
    nx = max(int(math.sqrt(points)), 12)
    ny = max(points // nx, 12)
    step = 20000.0 / math.sqrt(500000.0)
    ii, jj = (a.ravel() for a in np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij"))
    inner = (ii > 0) & (ii < nx - 1) & (jj > 0) & (jj < ny - 1)
    x = step * (ii + inner * rng.uniform(-0.22, 0.22, nx * ny))
    y = step * (jj + inner * rng.uniform(-0.22, 0.22, nx * ny))
    order = meshgen._morton_order(x, y)
    node = np.empty(nx * ny, np.int32)
    node[order] = np.arange(nx * ny, dtype=np.int32)
    x, y = x[order].copy(), y[order].copy()
    grid = node.reshape(nx, ny)
    a, b, c, d = grid[:-1, :-1].ravel(), grid[1:, :-1].ravel(), grid[1:, 1:].ravel(), grid[:-1, 1:].ravel()

    def angle(p, q, r):   # at q
        ux, uy, vx, vy = x[p] - x[q], y[p] - y[q], x[r] - x[q], y[r] - y[q]
        return np.arctan2(np.abs(ux * vy - uy * vx), ux * vx + uy * vy)

    ac = angle(a, b, c) + angle(c, d, a) <= np.pi
    tri = np.concatenate([np.stack([a, b, np.where(ac, c, d)], 1), np.stack([np.where(ac, a, b), c, d], 1)]).astype(np.int32)
    tri = tri[meshgen._morton_order(x[tri].mean(axis=1), y[tri].mean(axis=1))]
    sx, sy = step * (nx - 1), step * (ny - 1)
    taper = np.clip((np.minimum(x, sx - x) / sx - 0.05) / 0.05, 0.0, 1.0)
    z = -5e-4 * x
    for _ in range(40):
        w, cx, cy = rng.uniform(0.01, 0.075) * sx, rng.uniform(0.0, sx), rng.uniform(0.0, sy)
        z += taper**2 * (3.0 - 2.0 * taper) * rng.uniform(0.5, 3.0) * np.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2.0 * w * w))
    nmat = len(m.materials)
    west, east = np.stack([grid[0, 1:], grid[0, :-1]], 1), np.stack([grid[-1, :-1], grid[-1, 1:]], 1)
    return dataclasses.replace(
        m, x=x, y=y, z=z, tri=tri, tri_mat=np.clip(rng.normal(nmat / 2, nmat / 6, len(tri)), 0, nmat - 1).astype(np.int32),
        edges=np.concatenate([west, east]), edge_string=np.repeat(np.array([nmat, nmat + 1], np.int32), ny - 1),
        node_string=np.full(nx * ny, m.node_string[0], np.int32), h0=2.0 - z, u0=np.zeros(nx * ny), v0=np.zeros(nx * ny))


def _member(k, lo, hi):
    """One basin of the ensemble: its own size, bathymetry and time step."""
    rng = np.random.Generator(np.random.PCG64(k))
    return _basin(int(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2), 1000 + k, float(rng.uniform(2.0, 5.0)))


def _channel(nx, ny):
    return meshgen.channel(nx=nx, ny=ny, length=10.0 * nx, width=10.0 * ny)


def _mesh(case):
    return _channel(case["nx"], case["ny"]) if case["mesh"] == "channel" else _basin(case["points"])


def _moving(m, rng):
    """Two successive time levels of a state in slow motion: long waves on the surface and a smooth
    current, fading out where the water is shallower than a metre, still where the bed is dry."""
    span = max(float(np.ptp(m.x)), float(np.ptp(m.y)))
    depth = float(np.median(m.h0))

    def field(phase):
        f = np.zeros(m.nnodes)
        for kx, ky, p, a in phase:
            f += a * np.sin(2 * np.pi * (kx * m.x + ky * m.y) / span + p)
        return f

    def waves(amp):
        return [(rng.uniform(-3, 3), rng.uniform(-3, 3), rng.uniform(0, 2 * np.pi), amp * rng.uniform(0.4, 1.0)) for _ in range(4)]

    wh, wu, wv = waves(0.0005 * depth), waves(0.005), waves(0.005)
    fade = np.clip(m.h0, 0.0, 1.0)
    levels = []
    for lag in (0.0, 0.02):
        move = lambda w: [(kx, ky, p - lag, a) for kx, ky, p, a in w]  # noqa: E731
        levels.append((m.h0 + fade * field(move(wh)), fade * (0.01 + field(move(wu))), fade * field(move(wv))))
    return levels


def _pinned(arrays):
    out = []
    for a in arrays:
        t = torch.empty(len(a), dtype=torch.float64, pin_memory=True).numpy()
        t[:] = a
        out.append(t)
    return tuple(out)


def _model(m, rng, precision="fp64"):
    """The mesh with the run's own roughness (a scale on every material's Manning n).  On the mixed
    path the Newton loop does the refining, and runs to a tighter residual."""
    f = float(rng.uniform(0.8, 1.25))
    strings = [dataclasses.replace(s, manning_n=s.manning_n * f) if s.kind == "mat" else s for s in m.strings]
    tol = min(m.params.tol_nonlin, 1e-8) if precision == "mixed" else m.params.tol_nonlin
    return dataclasses.replace(m, strings=strings, params=dataclasses.replace(m.params, tol_nonlin=tol))


def prepare(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    s = dict(kind=case["kind"], case=case)
    if case["kind"] == "engine":
        s["engine"] = SW2Engine(PRECISION[case["precision"]])
        s["solvers"], s["levels"], s["out"] = [], [], []
        for k in range(case["members"]):
            m = _model(_member(k, case["lo"], case["hi"]), rng)
            s["solvers"].append(SW2GPU(m, PRECISION[case["precision"]]))
            s["levels"].append([_pinned(lv) for lv in _moving(m, rng)])
            s["out"].append(_pinned([np.zeros(m.nnodes)] * 3))
        return s
    if case["kind"] == "solve":
        # the Jacobian of a step in motion, a solution of the size of a Newton increment
        m = _model(_mesh(case), rng)
        g = SW2GPU(m)
        for lvl, state in enumerate(_moving(m, rng)):
            g.set_state(lvl, *state)
        g.step()
        rp, col, val, _ = g.load()
        g.close()
        x = _solution(m, seed)
        row = np.repeat(np.arange(m.nnodes), np.diff(rp))
        rhs = np.zeros((m.nnodes, 3))
        np.add.at(rhs, row, np.einsum("kij,kj->ki", val, x.reshape(-1, 3)[col]))
        dev = torch.device("cuda", torch.cuda.current_device())
        s["nnodes"], s["nnzb"] = m.nnodes, len(col)
        s["buffers"] = [torch.from_numpy(a).to(dev) for a in (rp, col, val.reshape(-1), rhs.reshape(-1), np.zeros(3 * m.nnodes))]
        s["its"] = ctypes.c_int32()
        return s
    m = _model(_mesh(case), rng, case.get("precision", "fp64"))
    if case["kind"] == "transport":
        m = dataclasses.replace(m, strings=list(m.strings), series=list(m.series))
        edges = [k for k, st in enumerate(m.strings) if st.kind == "edge"]
        m.constituents = [Constituent(ref_conc=1.0, diffusion=[0.5] * len(m.materials),
                                      edge_bc={e: meshgen.const_series(m, float(rng.uniform(0.5, 2.0))) for e in edges})
                          for _ in range(case["constituents"])]
        span = max(float(np.ptp(m.x)), float(np.ptp(m.y)))
        s["conc"] = _pinned([1.0 + 0.5 * np.sin(6.0 * m.x / span + rng.uniform(0, 6)) * np.cos(5.0 * m.y / span)
                             for _ in range(case["constituents"])])
        g = SW2GPU(m)
        g.set_mass_tracking(True)
    else:
        band = case["solver"] == "band"
        g = SW2GPU(m, PRECISION[case["precision"]], precond=capi.SW2GPU_PREC_BAND if band else capi.SW2GPU_PREC_BJACOBI)
        if case["graphs"]:
            g.set_graphs(case["graphs"])
    s["g"] = g
    s["levels"] = [_pinned(lv) for lv in _moving(m, rng)]
    s["out"] = _pinned([np.zeros(m.nnodes)] * 3)
    s["t"] = 2.0 * m.dt
    return s


def _accepted(st):
    if st["status"] != 0:
        raise RuntimeError(f"a time step failed: {st}")


def run(s):
    if s["kind"] == "solve":
        rp, col, val, rhs, x = s["buffers"]
        p = [ctypes.c_void_p(t.data_ptr()) for t in s["buffers"]]
        rc = lib().sw2gpu_bcsr_solve_noalloc(s["nnodes"], s["nnzb"], *p, 1e-11, 0.0, 500, None, ctypes.byref(s["its"]))
        if rc != 0:
            raise RuntimeError(lib().sw2gpu_last_error().decode())
        return x
    if s["kind"] == "engine":
        for g, levels in zip(s["solvers"], s["levels"]):
            for lvl, state in enumerate(levels):
                g.set_state(lvl, *state)
            g.t = 2.0 * g.model.dt
            s["engine"].add(g, s["case"]["steps"])
        for done in s["engine"].run():
            _accepted(done)
        return [g.get_state(0, out=o) for g, o in zip(s["solvers"], s["out"])]
    g = s["g"]
    for lvl, state in enumerate(s["levels"]):
        g.set_state(lvl, *state)
    g.t = s["t"]
    if s["kind"] == "transport":
        for k, c in enumerate(s["conc"]):
            g.set_conc(k, 0, c)
            g.set_conc(k, 1, c)
        _accepted(g.step())
        for st in g.transport_step():
            _accepted(st)
        mass, flux = g.step_mass()
        return dict(state=g.get_state(0, out=s["out"]), conc=[g.get_conc(k) for k in range(len(s["conc"]))], mass=mass)
    for _ in range(s["case"]["steps"]):
        _accepted(g.step())
    return g.get_state(0, out=s["out"])


def _solution(m, seed):
    rng = np.random.Generator(np.random.PCG64([int(seed), 1]))
    span = max(float(np.ptp(m.x)), float(np.ptp(m.y)))
    x = np.zeros((m.nnodes, 3))
    for c, amp in enumerate((0.02, 0.02, 0.01)):
        x[:, c] = amp * (np.sin(9.0 * m.x / span + rng.uniform(0, 6)) * np.cos(8.0 * m.y / span + rng.uniform(0, 6))
                         + 0.1 * rng.standard_normal(m.nnodes))
    return x.reshape(-1)


def exact(case, seed):
    # the right-hand side of the linear solve was made from its solution; a Newton step's result
    # has no value that plain numpy gives
    return _solution(_mesh(case), seed) if case["kind"] == "solve" else None


def work(case):
    """Mesh and two time levels read, one level written; two Newton iterations, each a residual and
    its nine derivatives per triangle (about 700 operations each) and 20 products with the Jacobian."""
    if case["kind"] == "engine":
        ts = [_member(k, case["lo"], case["hi"]).nelems2d for k in range(case["members"])]
        steps = case["steps"]
    elif case["mesh"] == "channel":
        ts, steps = [2 * case["nx"] * case["ny"]], case.get("steps", 1)
    else:
        ts, steps = [2 * case["points"]], case.get("steps", 1)
    t = float(sum(ts))
    v = t / 2
    if case["kind"] == "solve":
        return {"bytes": 7 * 76 * v + 48 * v, "flops": 40 * 7 * 18 * v}
    k = case.get("constituents", 0)
    return {"bytes": steps * (73 * t + (24 + 48 + 24) * v + k * (24 * v)),
            "flops": steps * (2 * (10 * 700 * t + 20 * 7 * 18 * v) + k * (4 * 300 * t + 50 * 7 * 2 * v))}
