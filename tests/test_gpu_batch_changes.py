"""Changes of a batch's members between two i2g_batch_step calls (rock types, grid
lines and fields, markers, extras): a replayed graph and the fused strategy's table
follow them, bit for bit what each context gives stepped alone through the same calls."""
import ctypes as C

import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


def members():
    insts = [synth.make_instance(f"b{i}", n=n, k=k, nsteps=3, seed=5000 + i, r_disk=r, vmax=10.0 ** (-9.5 + 0.5 * i),
                                extra_modes=2) for i, (n, k, r) in enumerate([(31, 3, 120e3), (47, 5, 200e3), (23, 4, 80e3)])]
    for i in insts:
        i.grid = {k: i.grid[k] for k in ("vx", "vy", "pr")}
        i.eta[::17] = 0.0  # viscosities that the averaging finds
        for k in ("marka0", "markb0", "markll"):
            i.types[k][5] = 0.5
    return insts


def stretched(g):
    u = (g - g[0]) / (g[-1] - g[0])
    out = g[0] + (g[-1] - g[0]) * (u + 0.3 * np.sin(np.pi * u) ** 2 / np.pi)
    out[-1] = g[-1]
    return out


def change(kind, ms, inst):
    if kind == "types":
        t = abi.types_from_instance(inst)
        for k in range(50):
            t.markro[k] *= 1.5
            t.markcp[k] += 7.0
        t.markim[7] = 1
        ms._check(ms.lib.i2g_set_types(ms.h, C.byref(t)), "types")
    elif kind == "lines":
        ms.set_grid(stretched(inst.gx), stretched(inst.gy), **inst.grid)
    elif kind == "field":
        ms.set_grid(inst.gx, inst.gy, **dict(inst.grid, mu=np.full(inst.nodenum, 1e19), exx=np.full(inst.nodenum, 1e-14)))
    elif kind == "markers":
        t = inst.mtype.copy()
        t[inst.mtype == 5], t[inst.mtype == 7] = 7, 6
        ms.set_markers(inst.x, inst.y, inst.T + 3.0, inst.eta, t)
    elif kind == "fewer":
        half = slice(0, inst.marknum // 2)
        ms.set_markers(inst.x[half], inst.y[half], inst.T[half], inst.eta[half], inst.mtype[half])
    elif kind == "extras":
        ms.set_marker_extras(tmax=inst.tmax, hi=np.full(inst.marknum, 0.5))
    elif kind == "porosity":
        ms.set_marker_extras(tmax=inst.tmax, por=np.full(inst.marknum, 0.2))


def outputs(steps):
    return [dict(ms.get_markers(), **{"node_" + k: v for k, v in ms.get_nodes().items()}) for ms in steps]


@pytest.mark.parametrize("kind", ["types", "lines", "field", "markers", "fewer", "extras", "porosity"])
@pytest.mark.parametrize("strategy,precision", [(abi.BATCH_STREAMS, abi.PREC_MIXED), (abi.BATCH_FUSED, abi.PREC_MIXED),
                                                (abi.BATCH_FUSED, abi.PREC_FP64)], ids=["graph", "fused-mixed", "fused-fp64"])
def test_member_changes_between_steps(kind, strategy, precision):
    insts = members()
    batched, alone = ([lib.MarkerStep.from_instance(i, precision=precision) for i in insts] for _ in range(2))
    for ms in alone:
        ms.set_fused(strategy == abi.BATCH_STREAMS)
    b = lib.Batch(batched)
    b.set_tune(strategy=strategy)
    dt = np.array([i.timestep for i in insts])
    ts = np.array([i.timesum for i in insts])
    for part in (0, 1):
        if part:
            for k in (0, 1):
                change(kind, batched[k], insts[k])
                change(kind, alone[k], insts[k])
        t0 = ts.copy()
        for _ in range(2):
            b.step(dt, ts, 2)
        b.sync()
        for k, ms in enumerate(alone):
            for s in range(4):
                ms.movemark(dt[k], t0[k])
                ms.ronurecalc(t0[k])
                t0[k] += dt[k]
    for got, want in zip(outputs(batched), outputs(alone)):
        for f in want:
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)
    b.close()


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
def test_single_precision_markers(precision):
    """The fused strategy keeps the positions of markers set in the reference's
    single-precision storage in that storage, as a context stepped alone does."""
    insts = members()
    fp = C.POINTER(C.c_float)

    def make(inst):
        ms = lib.MarkerStep.from_instance(inst, precision=precision, upload=False)
        ms.set_fused(False)
        ms.set_grid(inst.gx, inst.gy, **inst.grid)
        ms.set_nodes(**inst.nodes)
        f = [np.ascontiguousarray(a, dtype=np.float32) for a in (inst.x, inst.y, inst.T, inst.eta)]
        t = np.ascontiguousarray(inst.mtype, dtype=np.int8)
        assert ms.lib.i2g_set_markers_f32(ms.h, inst.marknum, *[a.ctypes.data_as(fp) for a in f],
                                          t.ctypes.data_as(C.c_char_p)) == 0
        ms.n = inst.marknum
        return ms
    for i in insts:
        i.scal["tmp_ambient"] = 150.1  # no single-precision number
    batched, alone = [make(i) for i in insts], [make(i) for i in insts]
    b = lib.Batch(batched)
    dt = np.array([i.timestep for i in insts])
    ts = np.array([i.timesum for i in insts])
    b.step(dt, ts, 3)
    b.sync()
    for ms, i in zip(alone, insts):
        ms.step(i.timestep, i.timesum, 3)
    for got, want in zip(outputs(batched), outputs(alone)):
        for f in want:
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)
    b.close()
