"""The marker step's workloads, each one pass through the public entry points.

A case is a dict of plain values; ``kind`` says which call sequence it is:

  steps       i2g_step (movemark + ronurecalc, several time steps), then the
              markers and the node fields into the caller's device arrays
  coupled     one time step as a host solver drives it: the solver's vx, vy, pr
              up, movemark, ronurecalc, the nine node fields down
  hosted      the drop-in's default: the host keeps the markers (single-precision
              storage) and hands them over and takes them back in every step
  thermal     movemark, ronurecalc, then titerate's marker temperature update
  adjoint     one iteration of an inversion: markers set, forward, backward
  batch       many planetesimals stepped side by side
  checkpoint  the output file's marker section written and read back

Shapes are the repository's own configurations (21^2, 101^2, 201^2, 401^2, 601^2,
1001^2 nodes, 3 x 3 to 6 x 6 markers per cell) and ragged ones between them.
Velocities are stream-function modes over the box, up to half a cell per step;
markers a jittered lattice (air, silicate, iron).  A pass on a state that is run
again goes back in time (the sign of the step, or of the velocity, alternates), so
that the markers stay distributed as they were.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from i2elvis_planet_b200 import abi, lib, synth

L_BOX = 500e3
R_DISK = 200e3
VMAX = 1e-9
TIMESUM = 1.0e6 * synth.SEC_PER_YEAR
NODES = synth.NODE_OUT
MARKERS = ("x", "y", "T", "eta", "p")


def _case(name, kind, nx, ny, k, steps=1, **more):
    c = dict(name=name, kind=kind, nx=nx, ny=ny, k=k, steps=steps, precision="mixed", uniform=True, order="cell",
             visc=False, table=False, instances=1)
    c.update(more)
    return c


def listed():
    return [
        # the smallest planetesimal, coupled to a host solver: launches and copies
        _case("coupled_21", "coupled", 21, 21, 4),
        # the reference's default host loop at the adjoint's grid: markers cross every step, FP64 form
        _case("hosted_201", "hosted", 201, 201, 4, precision="fp64"),
        # small, ordinary and largest grids of a run on the device, state read every 10 steps
        _case("steps_101", "steps", 101, 101, 4, 10),
        _case("steps_401", "steps", 401, 401, 4, 10),
        _case("steps_1001", "steps", 1001, 1001, 6, 10, order="random"),
        # refined (nonuniform), oblong, odd-sized grid with the rheology evaluated per marker
        _case("rheology_307x523", "steps", 307, 523, 5, 5, uniform=False, visc=True),
        # the bit-exact form
        _case("fp64_401", "steps", 401, 401, 4, 10, precision="fp64"),
        # the reference's default property model (densimod 2): P-T tables, melting
        _case("table_501", "steps", 501, 501, 5, 4, table=True),
        # a thermo-mechanical step with subgrid diffusion
        _case("thermal_601", "thermal", 601, 601, 4),
        # one iteration of an inversion: 20 steps forward, reverse sweep
        _case("adjoint_201", "adjoint", 201, 201, 4, 20),
        # an ensemble of planetesimals of different grids (101 to 401 lines)
        _case("batch_16", "batch", 101, 401, 4, 10, instances=16),
        # checkpoint and restart of a 401^2 run
        _case("checkpoint_401", "checkpoint", 401, 401, 4),
    ]


def draw(rng):
    kind = rng.choice(["steps"] * 5 + ["coupled", "hosted", "thermal", "adjoint", "batch", "checkpoint"])
    top = {"steps": 800, "coupled": 500, "hosted": 350, "thermal": 700, "adjoint": 240, "batch": 300,
           "checkpoint": 450}[kind]
    n = int(round(21 * (top / 21) ** rng.random()))
    ny = max(21, min(top, int(round(n * rng.choice([1.0, 1.0, 0.61, 1.47]))) + rng.randrange(3)))
    k = rng.randint(3, 6)
    c = _case("", kind, n, ny, k, rng.randint(2, 10), order=rng.choice(["cell", "random"]))
    del c["name"]
    if kind == "batch":
        c.update(nx=min(n, ny), ny=max(n, ny) + 1, instances=rng.randint(3, 16))
    elif kind == "steps":
        c["table"] = rng.random() < 0.25
        c["precision"] = "fp64" if not c["table"] and rng.random() < 0.3 else "mixed"
        c["visc"] = not c["table"] and rng.random() < 0.25
        c["uniform"] = rng.random() < 0.7
        if c["table"] or c["visc"] or c["precision"] == "fp64":  # dearer per step: no more than the largest listed
            c.update(nx=min(n, 500), ny=min(ny, 500), steps=min(c["steps"], 4))
    elif kind in ("coupled", "hosted"):
        c["precision"] = rng.choice(["mixed", "fp64"])
        c["steps"] = 1
    elif kind in ("thermal", "checkpoint"):
        c["steps"] = 1
    return c


def work(case):
    """Bytes: per step and marker x, y, T, eta, type read and x, y, p written, per
    node three fields read and eight written; the state read out once; the reverse
    sweep's checkpoints; host buffers once.  flops: the arithmetic of RK4 through
    the staggered grid, the property model and the sums."""
    b = f = 0.0
    for c in _members(case):
        nn, n, s, kind = c["nx"] * c["ny"], _count(c), c["steps"], c["kind"]
        b += s * (57.0 * n + 88.0 * nn)
        f += s * n * (220.0 + (150.0 if c["visc"] else 0.0) + (250.0 if c["table"] else 0.0))
        if kind in ("steps", "thermal", "batch"):
            b += 80.0 * n + 144.0 * nn
        if kind == "thermal":
            b += 66.0 * n + 48.0 * nn
            f += 90.0 * n
        if kind in ("coupled", "hosted"):
            b += 96.0 * nn + (33.0 * n if kind == "hosted" else 0.0)
        if kind == "adjoint":
            b += 33.0 * n + (-(-s // 5)) * 32.0 * n + 16.0 * n + 8 * 16.0 * nn
            f += s * n * 4 * (60.0 + 8 * 20.0)
        if kind == "checkpoint":
            b = 2 * (39.0 + 48.0) * n
            f = 20.0 * n
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ inputs
def _count(c):
    return (c["nx"] - 1) * (c["ny"] - 1) * c["k"] * c["k"]


def _members(case):
    """The instances of a batch: grids spread between nx and ny lines; else the case itself."""
    if case["kind"] != "batch":
        return [case]
    m = case["instances"]
    out = []
    for i in range(m):
        n = int(round(case["nx"] + (case["ny"] - case["nx"]) * ((i * 7) % m) / max(1, m - 1)))
        out.append(dict(case, nx=n, ny=n, k=3 + (i * 5 + case["k"]) % 4, instances=1))
    return out


def _lines(n, size, bend):
    t = np.linspace(0.0, 1.0, n)
    g = size * (t + bend * np.sin(2.0 * np.pi * t))
    g[0], g[-1] = 0.0, size
    return g


def _grid(c, seed):
    """Grid lines, velocity (unit-amplitude modes and their amplitudes), pressure, strain fields: host arrays."""
    r = np.random.default_rng(seed)
    nx, ny = c["nx"], c["ny"]
    xs, ys = L_BOX, L_BOX * (ny - 1) / (nx - 1)
    gx = _lines(nx, xs, 0.0 if c["uniform"] else 0.06)
    gy = _lines(ny, ys, 0.0 if c["uniform"] else -0.05)
    modes = [(1, 1)] + [tuple(int(v) for v in r.integers(1, 9, 2)) for _ in range(7 if c["kind"] == "adjoint" else 4)]
    amps = np.concatenate([[1.0], 0.3 * r.choice([-1.0, 1.0], len(modes) - 1)])
    mvx, mvy = synth.stream_velocity(gx, gy, modes, amps)
    vx, vy = amps @ mvx, amps @ mvy
    scale = VMAX / max(np.abs(vx).max(), np.abs(vy).max())
    g = dict(gx=gx, gy=gy, xs=xs, ys=ys, vx=vx * scale, vy=vy * scale, amps=amps * scale,
             dt=0.5 * min(np.diff(gx).min(), np.diff(gy).min()) / VMAX)
    if c["kind"] == "adjoint":
        g.update(mvx=mvx, mvy=mvy)
    ph = 2.0 * np.pi * r.random(2)
    xc, yc = np.concatenate([[0.0], 0.5 * (gx[1:] + gx[:-1])]), np.concatenate([[0.0], 0.5 * (gy[1:] + gy[:-1])])
    pr = 1e8 * (1.0 + 0.5 * np.outer(np.sin(2 * np.pi * xc / xs + ph[0]), np.cos(2 * np.pi * yc / ys + ph[1])))
    pr[0, :] = pr[:, 0] = 0.0
    g["fields"] = dict(vx=g["vx"], vy=g["vy"], pr=pr.reshape(-1))
    if c["table"]:
        g["fields"]["ga"] = np.full(nx * ny, 0.08)
    if c["visc"]:
        X, Y = np.meshgrid(gx / xs, gy / ys, indexing="ij")
        s = (np.sin(2 * np.pi * X + ph[0]) * np.cos(np.pi * Y)).reshape(-1)
        q = (np.cos(3 * np.pi * X) * np.sin(2 * np.pi * Y + ph[1])).reshape(-1)
        g["fields"].update(exx=1e-14 * s, eyy=-1e-14 * s, exy=3e-15 * q, sxx=2e7 * s, syy=-2e7 * s,
                           sxy=5e6 * q + 1e6)
    return g


def _markers(c, g, seed):
    """x, y, T, eta (FP64) and type (int8) on the GPU, in the caller's order."""
    gen = torch.Generator("cuda").manual_seed(seed)
    k, nc2 = c["k"], c["ny"] - 1
    n = _count(c)
    i = torch.arange(n, device="cuda")
    if c["order"] == "random":
        i = i[torch.randperm(n, generator=gen, device="cuda")]
    u = lambda: torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)  # noqa: E731
    cell, sub = i // (k * k), i % (k * k)
    gx, gy = (torch.from_numpy(g[a]).cuda() for a in ("gx", "gy"))
    m1, m2 = cell // nc2, cell % nc2
    x = gx[m1] + (gx[m1 + 1] - gx[m1]) * ((sub // k).double() + u()) / k
    y = gy[m2] + (gy[m2 + 1] - gy[m2]) * ((sub % k).double() + u()) / k
    del i, cell, sub, m1, m2
    r = torch.hypot(x - g["xs"] / 2, y - g["ys"] / 2)
    w = u()
    mt = torch.where(r > R_DISK, 0, torch.where(w < 0.2, 7, 5)).to(torch.int8)
    eta = torch.where(mt == 0, 1e18, torch.where(mt == 5, 1e20, 1e19)).double()
    eta = (eta * 10.0 ** torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)).clamp(1e18, 1e24)
    T = 150.0 + 1650.0 * torch.erf((R_DISK - r).clamp(min=0.0) / (R_DISK / 2))
    if c["table"]:
        # dry and wet silicate, crust and their molten types; wet markers around the ice's melting range
        w = u()
        sil = mt == 5
        for lo, hi, t in ((0.0, 0.25, 6), (0.25, 0.35, 11), (0.35, 0.40, 12), (0.40, 0.55, 25), (0.55, 0.62, 26),
                          (0.62, 0.68, 31), (0.68, 0.72, 32)):
            mt[sil & (w >= lo) & (w < hi)] = t
        T = torch.where((mt == 6) & (u() < 0.4), 262.0 + 30.0 * u(), T)
    return dict(x=x, y=y, T=T, eta=eta, type=mt)


def _setup(c):
    """Rock types, scalars and switches (synth's defaults, with the rheology or the table path on)."""
    types, markim = synth.default_types()
    flags, scal = synth.default_flags(), synth.default_scal()
    if c["visc"]:
        # power law with P-T dependence and brittle limit; P-T dependent Newtonian with Peierls creep; constant
        for t, v in ((5, dict(marknu=3.98e16, markdh=5.32e5, markdv=0.8, markss=3e7, markmm=3.5, markll=1.0,
                              marka0=1e8, markb0=0.3, marks1=9.1e9)),
                     (7, dict(marknu=1.26e11, markdh=5.32e5, markdv=0.1, marks0=6.3e-5, marks1=9.1e9)),
                     (0, dict(marknu=1e19))):
            for name, val in v.items():
                types[name][t] = val
    if c["table"]:
        flags["densimod"] = 2
        for t in (5, 6, 11, 12, 25, 26, 31, 32):
            for name, val in dict(markro=3300.0 if t % 20 in (5, 6) else 2900.0, markbb=3e-5, markaa=2e-5,
                                  markkt=3.0 if t < 20 else 2.0, markkf=150.0, markkp=2e-6,
                                  marknu=1e20 if t < 20 else 1e2, markn0=1e17 if t < 20 else 10.0).items():
                types[name][t] = val
        scal["core_form_time"] = 0.0
        scal["eps21"] = 0.5
    return types, markim, flags, scal


_TABLES = {}


def _table():
    if not _TABLES:
        _TABLES["td"] = synth.td_table(4242)
    return _TABLES["td"]


def _context(c, g, markers):
    e = np.empty(0)
    types, markim, flags, scal = _setup(c)
    inst = synth.Instance(name="case", xnumx=c["nx"], ynumy=c["ny"], xsize=g["xs"], ysize=g["ys"], gx=g["gx"],
                          gy=g["gy"], grid={}, nodes={}, x=e, y=e, T=e, eta=e, mtype=e, hi=e, por=e, tmax=e,
                          types=types, markim=markim, timestep=g["dt"], timesum=TIMESUM, nsteps=c["steps"],
                          mnumx=c["k"], mnumy=c["k"], flags=flags, scal=scal, td=_table() if c["table"] else None)
    prec = abi.PREC_MIXED if c["precision"] == "mixed" else abi.PREC_FP64
    ms = lib.MarkerStep.from_instance(inst, precision=prec, max_markers=_count(c), upload=False)
    ms.set_grid(g["gx"], g["gy"], **g["fields"])
    _set_dev(ms, markers)
    return ms


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _set_dev(ms, m):
    torch.cuda.current_stream().synchronize()  # the arrays are torch's work, the context has a stream of its own
    ms._check(ms.lib.i2g_set_markers_dev(ms.h, m["x"].numel(), *[_ptr(m[k]) for k in ("x", "y", "T", "eta", "type")]),
              "i2g_set_markers_dev")
    ms.n = m["x"].numel()


def _pinned(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def prepare(case, seed):
    seed = int(seed)
    mem = _members(case)
    S = dict(case=case, sign=1.0, time=TIMESUM)
    made = []
    for i, c in enumerate(mem):
        g = _grid(c, seed * 1000 + i)
        m = _markers(c, g, seed * 1000 + i)
        made.append((c, g, m, _context(c, g, m)))
    c, g, m, ms = made[0]
    S.update(ms=ms, g=g, dt=g["dt"])
    kind = c["kind"]
    n, nn = sum(_count(q) for q in mem), sum(q["nx"] * q["ny"] for q in mem)
    if kind in ("steps", "thermal", "batch"):
        S["out"] = {f: torch.empty(n, dtype=torch.float64, device="cuda") for f in MARKERS}
        S["out"].update({"n_" + f: torch.empty(nn, dtype=torch.float64, device="cuda") for f in NODES})
        a = b = 0
        S["read"] = []
        for q, _, _, ctx in made:
            S["read"].append((ctx, _count(q), [C.c_void_p(S["out"][f].data_ptr() + 8 * a) for f in MARKERS],
                              [C.c_void_p(S["out"]["n_" + f].data_ptr() + 8 * b) for f in NODES]))
            a, b = a + _count(q), b + q["nx"] * q["ny"]
    if kind == "batch":
        S["ctx"] = [q[3] for q in made]
        S["batch"] = lib.Batch(S["ctx"])
        S["batch"].set_tune(strategy=abi.BATCH_STREAMS)
        S["dts"] = np.array([q[1]["dt"] for q in made])
        S["times"] = np.full(len(made), TIMESUM)
    elif kind == "coupled":
        S["back"] = dict(g["fields"], vx=-g["vx"], vy=-g["vy"])
    elif kind == "hosted":
        S["host"] = {f: _pinned(m[f].float()) for f in ("x", "y", "T", "eta")}
        S["host"]["type"] = _pinned(m["type"])
        S["host"]["p"] = _pinned(torch.zeros(n))
        S["nodes"] = [_pinned(torch.zeros(nn, dtype=torch.float64)) for _ in NODES]
        S["up"] = [_pinned(torch.from_numpy(g["fields"][f])) for f in ("vx", "vy", "pr")]
    elif kind == "thermal":
        S["tk"] = [torch.from_numpy(a).cuda() for a in _solve(c, g)]
        torch.cuda.synchronize()
    elif kind == "adjoint":
        S["markers"] = m
        S["target"] = _target(c, g)
        ms.adjoint_setup(g["mvx"], g["mvy"])
    elif kind == "checkpoint":
        r = np.random.default_rng(seed)
        S["gr"], S["acc"] = (_pinned(torch.from_numpy(r.random(n, dtype=np.float32))) for _ in range(2))
        S["file"] = _pinned(torch.zeros(abi.PRN_RECORD_BYTES * n, dtype=torch.uint8))
    return S


def _solve(c, g):
    """Node temperatures before and after a heat solve."""
    X, Y = np.meshgrid(g["gx"] - g["xs"] / 2, g["gy"] - g["ys"] / 2, indexing="ij")
    r = np.hypot(X, Y)
    old = 150.0 + 1650.0 * np.tanh(np.maximum(0.0, R_DISK - r) / (R_DISK / 2))
    new = old + 40.0 * (np.sin(2 * np.pi * X / g["xs"] + 0.3) * np.cos(np.pi * Y / g["ys"]) + 0.25)
    return old.reshape(-1).copy(), new.reshape(-1).copy()


def _target(c, g):
    return _solve(c, g)[1]


# ------------------------------------------------------------------ one pass
def _read(S):
    for ctx, n, mk, nd in S["read"]:
        ctx._check(ctx.lib.i2g_get_markers_dev(ctx.h, n, *mk), "i2g_get_markers_dev")
        ctx._check(ctx.lib.i2g_get_nodes_dev(ctx.h, *nd), "i2g_get_nodes_dev")
    return S["out"]


def _f32(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


def run(S):
    c, ms, g = S["case"], S["ms"], S["g"]
    kind, dt = c["kind"], S["sign"] * S["dt"]
    if kind == "steps":
        ms.step(dt, S["time"], c["steps"], update_visc=c["visc"])
        S["time"] += c["steps"] * dt
        S["sign"] = -S["sign"]
        return _read(S)
    if kind == "thermal":
        old, new = S["tk"] if S["sign"] > 0 else S["tk"][::-1]
        ms.movemark(dt, S["time"])
        ms.ronurecalc(S["time"])
        ms.titerate_markers_dev(new, old, 1.0, S["dt"])
        S["sign"] = -S["sign"]
        return _read(S)
    if kind == "coupled":
        f = g["fields"] if S["sign"] > 0 else S["back"]
        ms.set_grid(g["gx"], g["gy"], **f)
        ms.movemark(S["dt"], S["time"])
        ms.ronurecalc(S["time"])
        S["time"] += S["dt"]
        S["sign"] = -S["sign"]
        return ms.get_nodes()
    if kind == "hosted":
        h, d, L = S["host"], abi.dptr, ms.lib
        n = h["x"].size
        t8 = h["type"].ctypes.data_as(C.c_char_p)
        ms._check(L.i2g_set_grid(ms.h, d(g["gx"]), d(g["gy"]), *[d(a) for a in S["up"]], *[None] * 8), "i2g_set_grid")
        ms._check(L.i2g_set_markers_f32(ms.h, n, *[_f32(h[f]) for f in ("x", "y", "T", "eta")], t8),
                  "i2g_set_markers_f32")
        ms.movemark(dt, S["time"])
        ms.ronurecalc(S["time"])
        ms._check(L.i2g_get_markers_f32(ms.h, n, _f32(h["x"]), _f32(h["y"]), _f32(h["T"]), None, _f32(h["p"])),
                  "i2g_get_markers_f32")
        ms._check(L.i2g_get_nodes(ms.h, *[d(a) for a in S["nodes"]]), "i2g_get_nodes")
        S["sign"] = -S["sign"]
        return {"x": h["x"], "y": h["y"], "T": h["T"], "p": h["p"], **{"n_" + f: a for f, a in zip(NODES, S["nodes"])}}
    if kind == "batch":
        # always forward in time: an ensemble's step is replayed as long as its time step stays
        S["batch"].step(S["dts"], S["times"], c["steps"])
        S["batch"].sync()
        return _read(S)
    if kind == "adjoint":
        _set_dev(ms, S["markers"])
        tk = ms.adjoint_forward(g["amps"], c["steps"], S["dt"], TIMESUM, 5)
        dT, da = ms.adjoint_backward(tk - S["target"])
        return {"tk": tk, "dT": dT, "da": da}
    ms.write_prn(gr=S["gr"], acc=S["acc"], out=S["file"])
    back = ms.read_prn(S["file"])
    return {"file": S["file"], **back}


# ------------------------------------------------------------------ 64 bits, without the framework
def exact(case, seed):
    seed = int(seed)
    parts = []
    for i, c in enumerate(_members(case)):
        g = _grid(c, seed * 1000 + i)
        m = _markers(c, g, seed * 1000 + i)
        parts.append(_exact_one(c, g, m, seed))
    if case["kind"] != "batch":
        return parts[0]
    return {f: torch.cat([p[f] for p in parts]) for f in parts[0]}


def _exact_one(c, g, m, seed):
    kind = c["kind"]
    if kind == "checkpoint":
        r = np.random.default_rng(seed)
        gr, acc = (r.random(_count(c), dtype=np.float32).astype(np.float64) for _ in range(2))
        return {"file": None, "gr": gr, "acc": acc, "mg_old": None, "mg_time": acc}
    if kind == "hosted":
        m = {f: (v if f == "type" else v.float().double()) for f, v in m.items()}
    P = _Plain(c, g)
    if kind == "adjoint":
        T0 = m["T"].clone().requires_grad_(True)
        amps = torch.from_numpy(g["amps"]).cuda().requires_grad_(True)
        vx, vy = (amps @ torch.from_numpy(g[f]).cuda() for f in ("mvx", "mvy"))
        x, y = m["x"], m["y"]
        for _ in range(c["steps"]):
            x, y = P.advect(x, y, vx, vy, g["dt"])
        T = torch.where(m["type"] < 2, 150.0, T0)
        num, den = P.scatter(x, y, [T, torch.ones_like(T)])
        tk = torch.where(den > 0, num / torch.where(den > 0, den, 1.0), 0.0)
        gr = tk.detach() - torch.from_numpy(_target(c, g)).cuda()
        dT, da = torch.autograd.grad(tk, (T0, amps), gr)
        return {"tk": tk.detach(), "dT": dT, "da": da}
    with torch.no_grad():
        out = P.steps(m, g["dt"], c["steps"])
        if kind == "thermal":
            P.heat(out, *[torch.from_numpy(a).cuda() for a in _solve(c, g)], g["dt"])
    if kind == "coupled":
        return {f: out["n_" + f] for f in NODES}
    if kind == "hosted":
        return {f: v for f, v in out.items() if f != "eta"}
    return out


class _Plain:
    """The marker step in plain torch, FP64, no attention to order or speed."""

    def __init__(self, c, g):
        self.c, self.nx, self.ny = c, c["nx"], c["ny"]
        self.xs, self.ys = g["xs"], g["ys"]
        self.gx, self.gy = (torch.from_numpy(g[a]).cuda() for a in ("gx", "gy"))
        self.xm, self.ym = 0.5 * (self.gx[1:] + self.gx[:-1]), 0.5 * (self.gy[1:] + self.gy[:-1])
        self.f = {k: torch.from_numpy(v).cuda() for k, v in g["fields"].items()}
        self.types, _, _, self.scal = _setup(c)
        self.tab = {k: torch.from_numpy(v).cuda() for k, v in self.types.items()}
        self.nn = self.nx * self.ny

    @staticmethod
    def cell(g, x):
        return (torch.searchsorted(g, x.detach().contiguous(), right=True) - 1).clamp(0, g.numel() - 2)

    def bil(self, fields, a, b, wx, wy):
        i = a * self.ny + b
        return [(1 - wx) * ((1 - wy) * f[i] + wy * f[i + 1]) + wx * ((1 - wy) * f[i + self.ny] + wy * f[i + self.ny + 1])
                for f in fields]

    def place(self, x, y):
        """Clamped point, its cell, basic weights."""
        x, y = x.clamp(0.0, self.xs), y.clamp(0.0, self.ys)
        a, b = self.cell(self.gx, x), self.cell(self.gy, y)
        return x, y, a, b, (x - self.gx[a]) / (self.gx[a + 1] - self.gx[a]), (y - self.gy[b]) / (self.gy[b + 1] - self.gy[b])

    def velocity(self, x, y, vx, vy):
        x, y, a, b, wx, wy = self.place(x, y)
        s = (b - (y.detach() < self.ym[b]).long()).clamp(0, self.ny - 3)
        u, = self.bil([vx], a, s, wx, (y - self.ym[s]) / (self.ym[s + 1] - self.ym[s]))
        s = (a - (x.detach() < self.xm[a]).long()).clamp(0, self.nx - 3)
        v, = self.bil([vy], s, b, (x - self.xm[s]) / (self.xm[s + 1] - self.xm[s]), wy)
        return u, v

    def centre(self, x, y, names):
        """Cell-centre fields at the markers."""
        x, y, a, b, _, _ = self.place(x, y)
        a = (a + (x > self.xm[a]).long()).clamp(1, self.nx - 2)
        b = (b + (y > self.ym[b]).long()).clamp(1, self.ny - 2)
        return self.bil([self.f[k] for k in names], a, b, (x - self.xm[a - 1]) / (self.xm[a] - self.xm[a - 1]),
                        (y - self.ym[b - 1]) / (self.ym[b] - self.ym[b - 1]))

    def advect(self, x, y, vx, vy, dt):
        k1x, k1y = self.velocity(x, y, vx, vy)
        k2x, k2y = self.velocity(x + k1x * dt / 2, y + k1y * dt / 2, vx, vy)
        k3x, k3y = self.velocity(x + k2x * dt / 2, y + k2y * dt / 2, vx, vy)
        k4x, k4y = self.velocity(x + k3x * dt, y + k3y * dt, vx, vy)
        return x + dt * (k1x + 2 * k2x + 2 * k3x + k4x) / 6, y + dt * (k1y + 2 * k2y + 2 * k3y + k4y) / 6

    def scatter(self, x, y, values):
        """Node sums of value x bilinear weight."""
        _, _, a, b, wx, wy = self.place(x, y)
        out = [torch.zeros(self.nn, dtype=torch.float64, device="cuda") for _ in values]
        for p in (0, 1):
            for q in (0, 1):
                w = (wx if p else 1 - wx) * (wy if q else 1 - wy)
                i = (a + p) * self.ny + b + q
                out = [o.index_add(0, i, w * v) for o, v in zip(out, values)]
        return out

    def viscosity(self, m, pb):
        """viscalc: power law, Newtonian, brittle and Peierls limits."""
        x, y = m["x"], m["y"]
        exx, sxx, eyy, syy = self.centre(x, y, ("exx", "sxx", "eyy", "syy"))
        xc, yc, a, b, _, _ = self.place(x, y)
        a, b = a.clamp(1, self.nx - 3), b.clamp(1, self.ny - 3)
        exy, sxy = self.bil([self.f["exy"], self.f["sxy"]], a, b, (xc - self.gx[a]) / (self.gx[a + 1] - self.gx[a]),
                            (yc - self.gy[b]) / (self.gy[b + 1] - self.gy[b]))
        e, s = ((0.5 * (u * u + v * v) + w * w).sqrt() for u, v, w in ((exx, eyy, exy), (sxx, syy, sxy)))
        rii = torch.where(m["eta"] > 0, (0.5 * s / e / m["eta"]) ** 0.87, 1.0)
        out = m["eta"].clone()
        for t in (0, 5, 7):
            T = {k: float(v[t]) for k, v in self.types.items()}
            k = m["type"] == t
            tk, p, eii, sii, ri = m["T"][k], pb[k], e[k], s[k], rii[k]
            z = torch.zeros_like(tk)
            sb = T["marka0"] + T["markb0"] * p * 1e5 * T["markll"]
            if T["marks0"] <= 0:
                sb = sb.clamp(max=T["marks1"])
            brit = z
            if T["markb0"] > 0 or T["marka0"] * T["markll"] > 0:
                brit = torch.where(eii > 0, torch.where(sb > 0, eii * ri / (0.5 * sb), 1.0 / T["markn0"]), z)
            pei = z
            rt = 8.314 * tk
            if T["marks0"] > 0:
                ok, s0 = (sii > 1e7) & (eii > 0), T["marks1"]
                q = torch.full_like(tk, s0 * 0.95)
                for _ in range(5):
                    q = (-rt / (T["markdh"] + T["markdv"] * p) * torch.log(eii / T["marks0"] / q / q)).sqrt()
                    q = (1.0 - torch.where(q > 1.0, -q, q)) * s0
                pei = torch.where(ok, eii / (0.5 * q.clamp(max=s0)), z)
            if T["markdh"] == 0 and T["markdv"] == 0:
                duct = torch.full_like(tk, 1.0 / T["marknu"])
            else:
                f = torch.exp(((T["markdh"] + T["markdv"] * p) / rt).clamp(max=150.0))
                if T["markss"] == 0 or T["markmm"] == 1.0:
                    duct = 1.0 / (T["marknu"] * f)
                else:
                    duct = 1.0 / (0.5 * T["marknu"] / T["markss"] ** (T["markmm"] - 1.0) * f)
                    duct = duct + torch.where(eii > 0, eii / (0.5 * (T["marknu"] * f * eii) ** (1.0 / T["markmm"])), z)
            n = torch.maximum(torch.maximum(duct, brit), pei)
            n = 1.0 / torch.where(n <= 0, 1.0 / T["markn1"], n)
            out[k] = n.clamp(T["markn0"], T["markn1"]).clamp(self.scal["nubeg"], self.scal["nuend"])
        return torch.where(m["T"] > 0, out, m["eta"])

    def steps(self, m, dt, nsteps):
        m = {k: v.clone() for k, v in m.items()}
        node = {f: torch.zeros(self.nn, dtype=torch.float64, device="cuda") for f in NODES}
        t, melt = TIMESUM, self.scal["eps21"]
        for _ in range(nsteps):
            m["p"], = self.centre(m["x"], m["y"], ("pr",))
            if self.c["visc"]:
                m["eta"] = self.viscosity(m, m["p"] * 1e-5)
            m["x"], m["y"] = self.advect(m["x"], m["y"], self.f["vx"], self.f["vy"], dt)
            melt = self.average(m, node, t, melt)
            t += dt
        return {**{f: m[f] for f in MARKERS}, **{"n_" + f: v for f, v in node.items()}}

    def average(self, m, node, t, melt):
        x, y, mt = m["x"], m["y"], m["type"].long()
        m["T"] = torch.where(mt < 2, self.scal["tmp_ambient"], m["T"])
        tk, tab = m["T"], self.tab
        ro, cp, kt = tab["markro"][mt], tab["markcp"][mt], tab["markkt"][mt].clone()
        bb, nu = torch.zeros_like(tk), m["eta"]
        r2 = (x - self.xs / 2) ** 2 + (y - self.ys / 2) ** 2
        nu = torch.where(r2.sqrt() > 0.95 * self.xs / 2, 1e22, nu)
        if self.c["table"]:
            ro, cp, kt, bb, nu, melt = self.melting(m, mt, nu, melt)
        kt = kt.clamp(0.001, self.scal["k_cutoff"])
        ht = torch.zeros_like(tk)
        for kinds, h in zip(((5, 6, 25, 26), (7, 8, 9, 10, 17, 18, 19)), _heat(t, self.scal)):
            for q in kinds:
                ht = torch.where(mt == q, h * ro, ht)
        w, *s = self.scatter(x, y, [torch.ones_like(tk), ro, bb, cp, kt, ht, tk])
        for f, v in zip(("ro", "et", "cp", "kt", "ht", "tk"), s):
            node[f] = torch.where(w != 0, v / w, node[f])
        _, _, a, b, wx, wy = self.place(x, y)
        lnu = torch.log(nu)
        q = 4 * (wx - 0.5).abs() * (wy - 0.5).abs()
        at = (a + (wx > 0.5)) * self.ny + b + (wy > 0.5)
        lo = self.viscous(node, "nu", at, q, lnu)
        q = 4 * (0.5 - (wx - 0.5).abs()) * (0.5 - (wy - 0.5).abs())
        lo = torch.minimum(lo, self.viscous(node, "nd", (a + 1) * self.ny + b + 1, q, lnu))
        for f in ("nu", "nd"):  # the contrast clamp reaches nodes without markers too
            node[f] = torch.minimum(torch.maximum(node[f], lo), lo * self.scal["nucontr"])
        return melt

    def viscous(self, node, f, at, q, lnu):
        z = torch.zeros(self.nn, dtype=torch.float64, device="cuda")
        w, s = z.index_add(0, at, q), z.index_add(0, at, q * lnu)
        v = torch.exp(s / w).clamp(self.scal["nubeg"], self.scal["nuend"])
        node[f] = torch.where(w != 0, v, node[f])
        return v[w != 0].min()

    def heat(self, out, old, new, dt):
        """titerate's marker part: subgrid diffusion, the node change, antidiffusion."""
        x, y, T = out["x"], out["y"], out["T"]
        _, _, a, b, wx, wy = self.place(x, y)
        to, tn, kt, cp, ro = self.bil([old, new, out["n_kt"], out["n_cp"], out["n_ro"]], a, b, wx, wy)
        d = (self.gx[a + 1] - self.gx[a]) ** -2 + (self.gy[b + 1] - self.gy[b]) ** -2
        ch = (to - T) * -torch.expm1((-kt / ro / cp * 2.0 * d * dt).clamp(min=-150.0))
        w, s = self.scatter(x, y, [torch.ones_like(T), ch])
        s = torch.where(w != 0, s / torch.where(w != 0, w, 1.0), s)
        back, = self.bil([s], a, b, wx, wy)
        out["T"] = T + ch + (tn - to) - back

    # densimod 2: tdbasecalc and meltpart1 for the table types, dencalc for the others
    def curve(self, p, crust):
        """Solidus and liquidus: Herzberg et al. (peridotite), Schmidt and Poli with Hess (crust)."""
        co = (1143.04342 + 273.15, 58.2946423e-4, 52.3439318e-8, -16.3201032e-12, 2.29886314e-16, -0.180865486e-20,
              0.00815679773e-24, -0.000197104325e-28, 1.97908526e-38)
        s = torch.zeros_like(p)
        for v in reversed(co):
            s = s * p + v
        s = torch.where(p < 21.5e4, s, 273.15 + 2157.5 + 11.7297e-4 * (p - 21.5e4))
        km = p * 3e-3
        sc = torch.where(km < 48.0, 972.6 - 2111.0 / (km + 10.63) + 70033.0 / (km + 10.63) ** 2,
                         935.4 + 0.1162 * km + 0.006937 * km * km)
        tl = torch.where(crust, 1423.15 + 3.5 * km, 1973.0 + 28.57e-4 * p)
        ts = torch.minimum(torch.where(crust, sc, s), tl - 100.0)
        return ts, tl

    def fraction(self, tk, p, crust):
        ts, tl = self.curve(p, crust)
        return ((tk - ts) / (tl - ts)).clamp(0.0, 1.0)

    @staticmethod
    def ice(tk, p):
        """Water ice (Dunaeva et al.), 10 K between onset and full melting; melt fraction."""
        lg, sq = torch.log(p), torch.sqrt(p)
        ts = torch.zeros_like(p)
        lo = 0.0
        for hi, k in ((2085.66, (273.0159, -0.0132, -0.1577, 0.0, 0.1516)), (3501.0, (10.277, 0.0265, 50.1624, 0.5868, -4.3288)),
                      (6324.0, (5.0321, -0.0004, 30.9482, 1.0018, 0.0)), (22160.0, (4.2804, -0.0013, 21.8756, 1.0018, 1.0785)),
                      (4e5, (-1355.42, 0.0018, 167.0609, -0.6633, 0.0)), (9e5, (0.2524, 0.0019, 0.2795, 0.5, 1.1675))):
            v = k[0] + k[1] * p + k[2] * lg + k[3] / p + k[4] * sq
            ts = torch.where((p >= lo) & (p < hi), v, ts)
            lo = hi
        return torch.where((p >= 0) & (p < 9e5), ((tk - ts) / 10.0).clamp(0.0, 1.0), 0.0)

    def melting(self, m, mt, nu, melt):
        tab, tk = self.tab, m["T"]
        pr, ga = self.centre(m["x"], m["y"], ("pr", "ga"))
        p = pr * 1e-5
        td = _table()
        istab = torch.zeros_like(mt, dtype=torch.bool)
        for t in (5, 6, 11, 12, 25, 26, 31, 32):
            istab |= mt == t
        crust = (mt == 11) | (mt == 12) | (mt == 31) | (mt == 32)
        # the other types
        ro = tab["markro"][mt] * (1 - tab["markbb"][mt] * (tk - 298.15)) * (1 + tab["markaa"][mt] * (p - 1) * 1e-3)
        bb = tab["markbb"][mt] / (1 - tab["markbb"][mt] * (tk - 298.15))
        cp, kt = tab["markcp"][mt], (tab["markkt"][mt] + tab["markkf"][mt] / (tk + 77.0)) * torch.exp(tab["markkp"][mt] * p)
        # the table
        low = p < 235000.0
        k1 = torch.where(low, (1.878 + 770.9 / tk.clamp(max=1200.0)) * (1 + 4.26e-6 * p),
                         (1.291 + 1157.0 / tk.clamp(max=2100.0)) * (1 + 2.5e-6 * p))
        k1 = k1 + torch.where(low, (tk / 1774.0) ** 3, (tk / 2117.0) ** 3)
        e = ((tk - td["tkmin"]) / td["tkstp"]).clamp(0.0, td["tknum"] - 1.0)
        n = ((p - td["pbmin"]) / td["pbstp"]).clamp(0.0, td["pbnum"] - 1.0)
        i, j = e.long().clamp(max=td["tknum"] - 2), n.long().clamp(max=td["pbnum"] - 2)
        e, n = e - i, n - j
        A = torch.from_numpy(td["td"]).cuda()
        db = crust.long()
        R = [A[i + u, j + v, db, 0] * 1000.0 for u in (0, 1) for v in (0, 1)]
        H = [A[i + u, j + v, db, 1] * 4183.7 for u in (0, 1) for v in (0, 1)]
        r = (R[0] * (1 - n) + R[1] * n) * (1 - e) + (R[2] * (1 - n) + R[3] * n) * e
        h = (((H[2] - H[0]) * (1 - n) + (H[3] - H[1]) * n) / td["tkstp"]).clamp(1e2, 5e4)
        q = 1e5 * td["pbstp"]
        x = (2 / (R[1] + R[0]) - (H[1] - H[0]) / q) * (1 - e) + (2 / (R[3] + R[2]) - (H[3] - H[2]) / q) * e
        x = (x * r / tk).clamp(-1e-2, 1e-2)
        xm = self.fraction(tk, p, crust)
        nt = torch.where((xm > 0) & (mt < 20), mt + 20, torch.where((xm <= 0) & (mt > 20), mt - 20, mt))
        nt = torch.where(istab, nt, mt)
        mol = istab & (nt > 20)
        nb = (nt - 20).clamp(min=0)
        r = torch.where(mol, r * (1 - xm) + xm * tab["markro"][nt] * (1 - tab["markbb"][nt] * (tk - 298.15)) *
                        (1 + tab["markaa"][nt] * (p - 1) * 1e-3), r)
        v = tab["marknu"][nt] * torch.exp((2.5 + ((1 - xm) / xm.clamp(min=1e-30)) ** 0.48) * (1 - xm))
        v = torch.minimum(torch.maximum(v, tab["markn0"][nt]), tab["markn1"][nt]).clamp(self.scal["nubeg"], self.scal["nuend"])
        nu = torch.where(mol & (xm > 0.1), v, nu)
        k1 = torch.where(mol, (tab["markkt"][nt] + tab["markkf"][nt] / (tk + 77.0)) * torch.exp(tab["markkp"][nt] * p) * xm +
                         (tab["markkt"][nb] + tab["markkf"][nb] / (tk + 77.0)) * torch.exp(tab["markkp"][nb] * p) * (1 - xm), k1)
        part = mol & (xm > 0) & (xm < 1)
        lat, dp = torch.where(crust, 380000.0, 400000.0), p * 0.001
        x = x + torch.where(part, lat * (self.fraction(tk, p - dp, crust) - self.fraction(tk, p + dp, crust)) * r /
                            (tk * 2e5 * dp), 0.0)
        h = h + torch.where(part, lat * (self.fraction(tk + 1, p, crust) - self.fraction(tk - 1, p, crust)) / 2.0, 0.0)
        wet = istab & (nt == 6)
        xi = self.ice(tk, p)
        part = wet & (xi > 0) & (xi < 1)
        lat = 517000.0 * 0.3
        x = x + torch.where(part, lat * (self.ice(tk, p - dp) - self.ice(tk, p + dp)) * r / (tk * 2e5 * dp), 0.0)
        h = h + torch.where(part, lat * (self.ice(tk + 1, p) - self.ice(tk - 1, p)) / 2.0, 0.0)
        ro, cp, bb, kt = (torch.where(istab, u, w) for u, w in ((r, ro), (h, cp), (x, bb), (k1, kt)))
        # soft turbulence in molten rock: the melt fraction the table marker before left (markers in the caller's order)
        left = self.fraction(torch.where(part, tk - 1, tk), p, crust)
        idx = torch.where(istab, torch.arange(mt.numel(), device="cuda"), -1).cummax(0).values
        before = torch.cat([torch.full((1,), -1, dtype=torch.long, device="cuda"), idx[:-1]])
        xs = torch.where(before >= 0, left[before.clamp(min=0)], melt)
        fl = torch.where(xs > 0.6, 100.0, tab["markn0"][mt] * torch.exp(-172.69 * (xs - 0.4)))
        on = ((mt == 25) | (mt == 26)) & (xs >= 0.4)
        dT = (tk - tk[0]).abs()
        fx = 0.089 * tab["markkt"][mt] ** (2 / 3) * dT ** (4 / 3) * (ro * ro * tab["markbb"][mt] * ga * cp / fl) ** (1 / 3)
        soft = (fx / 0.089) ** 1.5 / (dT ** 2 * ro) * (tab["markbb"][mt] * ga * cp / nu) ** -0.5
        kt = torch.where(on & (fx > 0.0001), soft, torch.where(on | (mt == 7), tab["markkt"][mt], kt))
        kt = torch.where((mt == 5) | (mt == 6), tab["markkt"][mt], kt)
        m["type"] = nt.to(torch.int8)
        last = int(idx[-1])
        return ro, cp, kt, bb, nu, float(left[last]) if last >= 0 else melt


def _heat(t, scal):
    """Radiogenic heat per kg of silicate and iron at time t."""
    a = t / (365.25 * 24 * 3600)
    f = lambda v, r: v * math.exp(-a * r)  # noqa: E731
    si = f(1.89716e23 * scal["al2627_init"] * 4.999e-13 / 3.264e13, 9.6673e-7) + f(0.40689 * 1.43e-11, 4.9867e-10) + \
        f(2.99e-12, 9.8458e-10) + f(1.6e-12, 1.5541e-10) + f(1e-12, 4.9511e-11)
    fe = f(1.971e24 * scal["fe6056_init"] * 4.3451e-13 / 1.183e14, 2.666e-7) + f(0.090625 * 1.43e-11, 4.9867e-10)
    return si, fe
