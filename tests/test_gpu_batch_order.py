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


@pytest.mark.parametrize("every", [1, 8], ids=["sorted-between", "ranked-between"])
def test_members_know_that_replays_moved_them(every):
    """Temperature updates and averaging of the general path between replayed steps:
    the members' ranks and order are of the positions the replays left."""
    insts = [synth.make_instance(f"m{i}", n=n, k=3, nsteps=1, seed=700 + i, r_disk=150e3, vmax=10.0 ** (-9.0 + i), extra_modes=2)
             for i, n in enumerate((61, 41))]
    batched, alone = ([lib.MarkerStep.from_instance(i, precision=abi.PREC_MIXED) for i in insts] for _ in range(2))
    for ms in batched:
        ms.set_reorder_interval(every)
    b = lib.Batch(batched)
    b.set_tune(strategy=abi.BATCH_STREAMS)
    dt = np.array([i.timestep for i in insts])
    ts = np.array([i.timesum for i in insts])

    def between(ms, k, call):
        tk = insts[k].nodes["tk"] + 500.0 + 20.0 * np.sin(np.arange(insts[k].nodenum) + call)
        ones = np.ones(tk.size)
        ms.titerate_markers(tk + 3.0, tk, 1.0, dt[k], kt=3.0 * ones, cp=1000.0 * ones, ro=3300.0 * ones)
    for call in range(5):
        t = ts.copy()
        b.step(dt, ts, 2)
        for k, ms in enumerate(alone):
            for _ in range(2):
                ms.movemark(dt[k], t[k])
                ms.ronurecalc(t[k])
                t[k] += dt[k]
        for ms in (*batched, *alone):
            k = (batched.index(ms) if ms in batched else alone.index(ms))
            between(ms, k, call)
        if call == 4:  # the general path's averaging of the markers as they are
            for ms, k in zip((*batched, *alone), (0, 1, 0, 1)):
                ms.ronurecalc(t[k] + dt[k])
    for got, want in zip(batched, alone):
        for a, c in ((got.get_markers(), want.get_markers()), (got.get_nodes(), want.get_nodes())):
            for f in c:
                np.testing.assert_array_equal(a[f], c[f], err_msg=f)
    b.close()
