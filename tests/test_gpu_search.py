"""The cell search through an axis' bins and the stage walk on grids whose spacing
varies by 1, 20 and 5000 times, with markers on lines, on midpoints, next to them and
on the box: the FP64 form equals the oracle bit for bit (positions, pressure), the
mixed form's fused step moves every marker within 1e-6 of the smallest cell of it."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


def stretched(ratio, seed):
    inst = synth.make_instance("s", n=61, k=4, nsteps=2, seed=seed)
    for axis, size in (("gx", inst.xsize), ("gy", inst.ysize)):
        w = ratio ** np.abs(np.linspace(-1.0, 1.0, 60)) if axis == "gx" else ratio ** np.linspace(0.0, 1.0, 60)
        g = np.concatenate([[0.0], np.cumsum(w)])
        g *= size / g[-1]
        g[-1] = size
        setattr(inst, axis, g)
    mvx, mvy = synth.stream_velocity(inst.gx, inst.gy, inst.modes, inst.amps)
    inst.grid["vx"], inst.grid["vy"] = inst.amps @ mvx, inst.amps @ mvy
    cell = min(np.diff(inst.gx).min(), np.diff(inst.gy).min())
    inst.timestep = 0.5 * cell / max(np.abs(inst.grid["vx"]).max(), np.abs(inst.grid["vy"]).max())
    pick = np.arange(0, inst.marknum, 7)
    line = (pick * 13) % 61
    for arr, g in ((inst.x, inst.gx), (inst.y, inst.gy)):
        arr[pick] = g[line]
        mid = pick + 1
        mid = mid[mid < inst.marknum]
        m = np.minimum((mid * 5) % 61, 59)
        arr[mid] = (g[m] + g[m + 1]) / 2.0
        near = pick + 2
        near = near[near < inst.marknum]
        arr[near] = np.clip(np.nextafter(g[(near * 3) % 61], np.where(near % 2, 1e9, -1e9)), 0.0, g[-1])
    return inst


@pytest.mark.parametrize("ratio", [1.0, 20.0, 5000.0])
def test_search_on_stretched_grids(ratio):
    inst = stretched(ratio, 21)
    m64, n64, ms = lib.run_instance(inst, precision=abi.PREC_FP64)
    ms.close()
    ref = oracle.Oracle(inst).run(order=oracle.ORDER_CELL)
    for f in ("x", "y", "p"):
        np.testing.assert_array_equal(m64[f], getattr(ref, f), err_msg=f)
    mm, nm, ms = lib.run_instance(inst, precision=abi.PREC_MIXED)
    assert ms.fused_info()["fused_moves"] == 2
    ms.close()
    cell = min(np.diff(inst.gx).min(), np.diff(inst.gy).min())
    assert max(np.abs(mm["x"] - m64["x"]).max(), np.abs(mm["y"] - m64["y"]).max()) <= 1e-6 * cell
