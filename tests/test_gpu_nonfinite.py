"""FP64 form: an infinite node velocity carries a marker out of the box as the oracle
has it (an infinite position, the temperature reset), not to a NaN."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_infinite_velocity(sign):
    inst = synth.make_config("micro", nsteps=1)
    inst.grid["vx"] = np.zeros(inst.nodenum)
    inst.grid["vy"] = np.zeros(inst.nodenum)
    inst.grid["vx"][7 * inst.ynumy + 9] = sign * np.inf
    want = oracle.Oracle(inst).run(order=oracle.ORDER_CELL)
    ms = lib.MarkerStep.from_instance(inst, precision=abi.PREC_FP64)
    ms.movemark(inst.timestep, inst.timesum)
    got = ms.get_markers()
    ms.close()
    assert np.isinf(want.x).sum() > 10
    for f in ("x", "y", "T"):
        np.testing.assert_array_equal(got[f], getattr(want, f), err_msg=f)
