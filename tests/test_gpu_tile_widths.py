"""Every tile width of the averaging's cell sums gives the same nine node fields bit for
bit: a context alone, whose width follows from its grid, against the fused batch
strategy at 8, 16 and 32 cell columns."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [6, 40, 321])
def test_all_fields_at_every_width(n, precision):
    inst = synth.make_instance("s", n=n, k=2, nsteps=1, seed=31)
    alone = lib.MarkerStep.from_instance(inst, precision=precision)
    alone.set_fused(False)
    alone.step(inst.timestep, inst.timesum, 1)
    want = alone.get_nodes()
    alone.close()
    for cols in (8, 16, 32):
        ms = lib.MarkerStep.from_instance(inst, precision=precision)
        b = lib.Batch([ms])
        b.set_tune(tile_cols=cols)
        b.step(np.array([inst.timestep]), np.array([inst.timesum]), 1)
        b.sync()
        got = ms.get_nodes()
        b.close()
        ms.close()
        for k in synth.NODE_OUT:
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{cols} {k}")
