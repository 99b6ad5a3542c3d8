"""The adjoint of an RK4 step weights its stages with the quotients by 6 and 3.

A still marker on a velocity node sees one mode that is 1 there: its dL/da is dL/dx dt
for an Euler step, and for RK4 the sum of that over 6, 3, 3 and 6 in the reverse sweep's
order, in FP64 arithmetic to the bit.  (A second marker makes the temperature average
depend on where the first one is; the mode does not reach it.)"""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
def test_stage_weights_are_quotients(precision):
    n, i, j = 33, 12, 17
    base = synth.subset(synth.make_instance("s", n=n, k=1, nsteps=1, seed=4), np.arange(2))
    w = base.gx[1] - base.gx[0]
    base.x[:] = [i * w, (i - 0.25) * w]
    base.y[:] = [(j + 0.5) * w, (j - 0.625) * w]
    base.T[:], base.eta[:], base.mtype[:] = [700.0, 1100.0], 1e20, 5
    mode = np.zeros((1, base.nodenum))
    mode[0, i * n + j] = 1.0
    g = np.zeros(base.nodenum)
    g[i * n + j] = 1.0
    differ = 0
    for k in range(8):
        dt = 1e11 * (1 + synth.rng_uniform(9, k, 1)[0])
        da = []
        for markmod in (1, 2):
            inst = base.copy()
            inst.flags["markmod"] = markmod
            ms = lib.MarkerStep.from_instance(inst, precision=precision)
            ms.adjoint_setup(mode, np.zeros_like(mode))
            ms.adjoint_forward(np.zeros(1), 1, dt, inst.timesum, ckpt_every=1)
            da.append(ms.adjoint_backward(g)[1][0])
            ms.close()
        euler, rk4 = da
        assert euler != 0
        assert rk4 == ((euler / 6 + euler / 3) + euler / 3) + euler / 6
        differ += euler / 6 != euler * (1 / 6)
    assert differ
