"""The temperature update's cell sums (a thread per cell, four records in flight) at
numbers of cells around a block's 256 and markers per cell around the four: the FP64
form equals the oracle within exp's last bit (1e-13 of max |T|), the mixed form is
within 1e-6 of it."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(5, 1), (16, 2), (17, 3), (18, 1), (40, 2)])
def test_cell_sums_of_the_temperature_update(n, k):
    inst = synth.make_instance("t", n=n, k=k, nsteps=1, seed=13)
    f = synth.thermal_fields(inst, fluid_frac=0.05, cold_frac=0.02)
    tk_new, heatdif = f["tk_new"], 1.0
    o = oracle.Oracle(inst)
    s = o.initial_state()
    o.titerate_markers(s, tk_new, heatdif, inst.timestep, order=oracle.ORDER_CELL)
    T = {}
    for p in (abi.PREC_FP64, abi.PREC_MIXED):
        ms = lib.MarkerStep.from_instance(inst, precision=p)
        nd = inst.nodes
        ms.titerate_markers(tk_new, nd["tk"], heatdif, inst.timestep, kt=nd["kt"], cp=nd["cp"], ro=nd["ro"])
        T[p] = ms.get_markers(fields=("T",))["T"]
        ms.close()
    top = np.abs(s.T).max()
    assert np.abs(T[abi.PREC_FP64] - s.T).max() <= 1e-13 * top
    assert np.abs(T[abi.PREC_MIXED] - T[abi.PREC_FP64]).max() <= 1e-6 * top
