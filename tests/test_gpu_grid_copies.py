"""i2g_set_grid and i2g_get_nodes on both sides of the sizes where a small grid crosses
through the context's pinned memory: the same fields from pageable and from pinned
arrays, fields left out after a call that gave them, and a node read-out of some fields
only give the outputs of a fresh context bit for bit (copies only)."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


def step(inst, precision, calls):
    ms = lib.MarkerStep.from_instance(inst, precision=precision)
    for fields in calls:
        ms.set_grid(inst.gx, inst.gy, **fields)
    ms.movemark(inst.timestep, inst.timesum, update_visc=True)
    ms.ronurecalc(inst.timesum)
    mk, nodes = ms.get_markers(fields=("x", "y", "eta", "p")), ms.get_nodes()
    some = np.full(ms.nodenum, -7.0)
    ms._check(ms.lib.i2g_get_nodes(ms.h, None, None, None, None, None, None, None, abi.dptr(some), None), "nodes")
    np.testing.assert_array_equal(some, nodes["tk"])
    ms.close()
    return dict(mk, **{"node_" + k: v for k, v in nodes.items()})


def pinned(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n", [5, 21, 90, 91, 250])  # 64 KB fields at 90, 5 MB in all at 243
def test_small_grids_cross_in_one_copy(n, precision):
    inst = synth.make_instance("g", n=n, k=2, nsteps=1, seed=9)
    r = np.random.default_rng(n)
    full = {k: inst.grid[k] for k in ("vx", "vy", "pr")}
    for k in ("exx", "eyy", "exy"):
        full[k] = 1e-14 * r.standard_normal(n * n)
    for k in ("sxx", "syy", "sxy"):
        full[k] = 1e6 * r.standard_normal(n * n)
    few = {k: full[k] for k in ("vx", "vy", "pr")}
    for fields, before in ((full, few), (few, full)):
        one = step(inst, precision, [fields])
        for calls in ([before, fields], [{k: pinned(v) for k, v in fields.items()}]):
            two = step(inst, precision, calls)
            for k in one:
                np.testing.assert_array_equal(one[k], two[k], err_msg=k)
