"""i2g_set_grid between calls: other grid lines make the markers' cells and order anew
(the averaging and the temperature update that follow give what a fresh context with
those lines and markers gives, bit for bit)."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu
FORMS = pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])


def stretched(g, s):
    u = (g - g[0]) / (g[-1] - g[0])
    out = g[0] + (g[-1] - g[0]) * (u + s * np.sin(np.pi * u) ** 2 / np.pi)
    out[0], out[-1] = g[0], g[-1]
    return out


@FORMS
@pytest.mark.parametrize("before", ["set", "moved", "averaged", "sorted"])
def test_other_lines_before_averaging(before, precision):
    inst = synth.make_config("c1", permute=True)
    gx, gy = stretched(inst.gx, 0.4), stretched(inst.gy, -0.3)
    ms = lib.MarkerStep.from_instance(inst, precision=precision)
    ms.set_fused(False)
    ms.set_reorder_interval(1 if before == "sorted" else 8)
    if before != "set":
        ms.movemark(inst.timestep, inst.timesum)
    if before in ("averaged", "sorted"):
        ms.ronurecalc(inst.timesum)
    mk = ms.get_markers()
    fresh = lib.MarkerStep.from_instance(inst, precision=precision)
    fresh.set_fused(False)
    out = []
    for m in (ms, fresh):
        m.set_grid(gx, gy, **inst.grid)
        if m is fresh:
            m.set_markers(mk["x"], mk["y"], mk["T"], mk["eta"], inst.mtype)
        m.set_nodes(**inst.nodes)
        m.ronurecalc(inst.timesum)
        nodes = m.get_nodes()
        tk = inst.nodes["tk"] + 10.0 * np.sin(np.arange(inst.nodenum))
        m.titerate_markers(tk, inst.nodes["tk"], 1.0, inst.timestep)
        out.append((nodes, m.get_markers(fields=("x", "y", "T"))))
        m.close()
    for k in synth.NODE_OUT:
        np.testing.assert_array_equal(out[0][0][k], out[1][0][k], err_msg=k)
    for k in ("x", "y", "T"):
        np.testing.assert_array_equal(out[0][1][k], out[1][1][k], err_msg=k)
