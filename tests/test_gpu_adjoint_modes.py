"""The adjoint's mode sums at every register capacity (4, 8, 16 modes) and its edges."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nm,outgrid,markmod", [(1, 2, 2), (4, 2, 2), (5, 0, 2), (8, 1, 1), (9, 2, 2), (16, 2, 2)])
def test_mode_capacities(precision, nm, outgrid, markmod):
    """A mode's gradient does not depend on the modes set beside it: each mode next
    to the whole flow (capacity 4) against all of them together.  The two flows
    differ by the rounding of sum_m a_m v_m alone, 16 units in the last place at
    most, and the sums by their order: 1e-11 of the largest gradient."""
    base = synth.make_config("micro", extra_modes=7)
    base.flags["outgrid"], base.flags["markmod"] = outgrid, markmod
    rng = np.random.default_rng(nm)
    mvx, mvy = (np.concatenate([m, m[::-1] * 0.5])[:nm].copy() for m in (base.mode_vx, base.mode_vy))
    amps = base.amps[0] * rng.uniform(0.2, 1.0, nm)
    g = rng.standard_normal(base.nodenum)
    vx, vy = amps @ mvx, amps @ mvy

    def grad(mx, my, a):
        ms = lib.MarkerStep.from_instance(base, precision=precision)
        ms.adjoint_setup(mx, my)
        tk = ms.adjoint_forward(a, 7, base.timestep, base.timesum, 3)
        dT, da = ms.adjoint_backward(g)
        ms.close()
        return tk, dT, da

    tk, dT, da = grad(mvx, mvy, amps)
    # mode m alone: the whole flow as mode 0, mode m with amplitude 0
    for m in range(nm):
        tk1, dT1, da1 = grad(np.stack([vx, mvx[m]]), np.stack([vy, mvy[m]]), np.array([1.0, 0.0]))
        scale = np.abs(da).max()
        np.testing.assert_allclose(dT1, dT, rtol=0, atol=1e-11 * np.abs(dT).max())
        assert abs(da1[1] - da[m]) <= 1e-11 * scale, (m, da1[1], da[m])
    assert abs(da @ amps - da1[0]) <= 1e-11 * max(abs(da1[0]), np.abs(da * amps).sum())
