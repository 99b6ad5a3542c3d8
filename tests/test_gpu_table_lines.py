"""densimod 2, markers exactly at the table's temperatures: the heat capacity is the slope
of the cell that starts there in both forms (it jumps from cell to cell), the weights'
FP32 rounding apart."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


def test_table_lines_keep_their_cell():
    step, base = 49.0, 300.0  # (k 49) (1 / 49) < k for k = 1, 2, 3, 4, 6, ...
    inst = synth.with_table(synth.make_config("micro", nsteps=1))
    tk = base + step * np.arange(100)
    slope = np.where(np.arange(100) % 2 == 0, 1000.0, 2000.0)
    h = np.concatenate([[0.0], np.cumsum(slope[:-1] * step)]) / 4183.7 + 100.0
    td = np.zeros((100, 50, 2, 5))
    td[..., 0] = 3.3
    td[..., 1] = h[:, None, None]
    inst.td = dict(inst.td, td=td, tknum=100, pbnum=50, tkmin=base, pbmin=1.0, tkstp=step, pbstp=20000.0)
    inst.mtype[:] = 5
    inst.grid = dict(inst.grid, vx=np.zeros(inst.nodenum), vy=np.zeros(inst.nodenum))
    for k in (1, 2, 3, 4, 5, 6, 13):
        inst.T[:] = tk[k]
        cp = []
        for precision in (abi.PREC_FP64, abi.PREC_MIXED):
            ms = lib.MarkerStep.from_instance(inst, precision=precision)
            ms.movemark(inst.timestep, inst.timesum)
            ms.ronurecalc(inst.timesum)
            cp.append(ms.get_nodes()["cp"])
            ms.close()
        assert (np.abs(cp[0] / slope[k] - 1) < 1e-9).all()
        assert np.abs(cp[1] / cp[0] - 1).max() <= 1e-6, (k, np.abs(cp[1] / cp[0] - 1).max())
