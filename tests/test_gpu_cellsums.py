"""The cell sums' tile width (8, 16 or 32 cell columns by the grid's size): at sizes that
take each of the three, whole and with a remainder, the FP64 form's node fields equal
the oracle's in the same order bit for bit."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 40, 321, 513])  # 8, 8, 16 and 32 columns with 148 SMs
def test_tile_widths(n):
    inst = synth.make_instance("s", n=n, k=2, nsteps=1, seed=31)
    mk, nodes, ms = lib.run_instance(inst, precision=abi.PREC_FP64)
    ms.close()
    ref = oracle.Oracle(inst).run(order=oracle.ORDER_CELL)
    np.testing.assert_array_equal(mk["x"], ref.x)
    for k in ("ro", "et", "cp", "ht", "tk", "po"):
        np.testing.assert_array_equal(nodes[k], ref.nodes[k], err_msg=k)
