"""The streams strategy's replays run after what the contexts' own streams still hold:
the record moves at the end of the call before (every call here) and a caller's own
steps on a member, with no synchronisation between: bit for bit each context's steps
alone."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


def test_replays_wait_for_the_contexts_streams():
    insts = [synth.make_instance(f"o{i}", n=n, k=4, nsteps=1, seed=600 + i, r_disk=200e3, vmax=10.0 ** (-9.0 + i), extra_modes=2)
             for i, n in enumerate((201, 61))]
    batched, alone = ([lib.MarkerStep.from_instance(i, precision=abi.PREC_MIXED) for i in insts] for _ in range(2))
    for ms in batched:
        ms.set_reorder_interval(1)  # the fused step moves the records every fourth step
    b = lib.Batch(batched)
    b.set_tune(strategy=abi.BATCH_STREAMS)
    dt = np.array([i.timestep for i in insts])
    ts = np.array([i.timesum for i in insts])
    steps = 0
    for call in range(12):
        b.step(dt, ts, 4)
        steps += 4
        if call % 3 == 2:
            for k, ms in enumerate(batched):
                ms.movemark(dt[k], ts[k])
                ms.ronurecalc(ts[k])
            ts += dt
            steps += 1
    for got, ms, i in zip(batched, alone, insts):
        t = i.timesum
        for _ in range(steps):
            ms.movemark(i.timestep, t)
            ms.ronurecalc(t)
            t += i.timestep
        for a, c in ((got.get_markers(), ms.get_markers()), (got.get_nodes(), ms.get_nodes())):
            for f in c:
                np.testing.assert_array_equal(a[f], c[f], err_msg=f)
    b.close()
