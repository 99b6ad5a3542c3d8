"""A second averaging without a movemark between, after a call that moved the marker
records into cell order: on the table path the melt pass reads each marker's cell, so
every reorder interval has to give the same bits, which the calls that move nothing
(a long interval) define."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
def test_table_path_repeated_averaging(precision):
    inst = synth.with_table(synth.make_config("c1", permute=True))
    inst.scal["k_cutoff"] = 1e40  # the molten conductivities, which read the melt fractions, stay apart
    outs = []
    for every in (100, 1, 3, 8):
        ms = lib.MarkerStep.from_instance(inst, precision=precision)
        ms.set_reorder_interval(every)
        ms.set_marker_extras(tmax=inst.tmax)
        ts = inst.timesum
        for s in range(8):
            ms.movemark(inst.timestep, ts)
            ms.ronurecalc(ts, track_tmax=True)
            if s in (2, 4, 7):
                ms.ronurecalc(ts, track_tmax=True)
            ts += inst.timestep
        outs.append((ms.get_markers(fields=("x", "y", "T", "eta", "p", "type"), with_tmax=True), ms.get_nodes(),
                     ms.get_melt_state()))
        ms.close()
    m0, n0, e0 = outs[0]
    for mk, nodes, eps in outs[1:]:
        for f in mk:
            np.testing.assert_array_equal(mk[f], m0[f], err_msg=f)
        for k in synth.NODE_OUT:
            np.testing.assert_array_equal(nodes[k], n0[k], err_msg=k)
        np.testing.assert_array_equal(eps, e0)
