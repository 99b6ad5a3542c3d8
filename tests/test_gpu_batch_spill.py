"""A batch member whose cells overflow their buckets by a few records keeps them in the
overflow list while its step is replayed: the same bits as a context stepped alone,
which enlarges its buckets, and no wait for other work on the device."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


def gathering(lines, each, seed):
    """``each`` markers in three neighbouring cells of a row, the flow gathers all of
    them in the middle one: 3 x each records for a bucket of each + max(8, each / 2)."""
    inst = synth.subset(synth.make_instance("g", n=lines, k=2, nsteps=1, seed=seed), np.arange(3 * each))
    w = inst.gx[1] - inst.gx[0]
    c = (lines - 1) // 2
    u, v = synth.rng_uniform(seed, 1, 3 * each), synth.rng_uniform(seed, 2, 3 * each)
    inst.x[:] = (c - 1 + np.repeat(np.arange(3), each) + 0.02 + 0.96 * u) * w
    inst.y[:] = (c + 0.02 + 0.96 * v) * w
    inst.T[:] = 300.0 + 1000.0 * u
    inst.eta[:] = 10.0 ** (18 + 4 * v)
    inst.mtype[:] = np.where(u < 0.5, 5, 7)
    X = np.repeat(inst.gx, lines)
    inst.grid = dict(vx=-1.5 * (X - (c + 0.5) * w) / inst.timestep, vy=np.zeros(inst.nodenum), pr=inst.grid["pr"])
    return inst


@pytest.mark.parametrize("lines", [33, 193], ids=["two-lanes", "one-lane"])
@pytest.mark.parametrize("each", [9, 10, 61])
def test_small_spills_while_replayed(lines, each):
    insts = [gathering(lines, each, 5), synth.make_instance("p", n=41, k=3, nsteps=1, seed=6)]
    batched, alone = ([lib.MarkerStep.from_instance(i, precision=abi.PREC_MIXED) for i in insts] for _ in range(2))
    b = lib.Batch(batched)
    b.set_tune(strategy=abi.BATCH_STREAMS)
    dt = np.array([i.timestep for i in insts])
    ts = np.array([i.timesum for i in insts])
    t0 = ts.copy()
    for n in (1, 3, 2):
        b.step(dt, ts, n)
    b.sync()
    assert batched[0].fused_info()["bucket_growths"] == 0
    for k, ms in enumerate(alone):
        for _ in range(6):
            ms.movemark(dt[k], t0[k])
            ms.ronurecalc(t0[k])
            t0[k] += dt[k]
    assert alone[0].fused_info()["bucket_growths"] >= 1
    for got, want in zip(batched, alone):
        for a, c in ((got.get_markers(), want.get_markers()), (got.get_nodes(), want.get_nodes())):
            for f in c:
                np.testing.assert_array_equal(a[f], c[f], err_msg=f)
    b.close()


def test_spill_check_leaves_the_default_stream_alone():
    import torch
    insts = [gathering(33, 10, 5)]
    steps = [lib.MarkerStep.from_instance(i, precision=abi.PREC_MIXED) for i in insts]
    b = lib.Batch(steps)
    b.set_tune(strategy=abi.BATCH_STREAMS)
    dt, ts = np.array([insts[0].timestep]), np.array([insts[0].timesum])
    b.step(dt, ts, 2)
    b.sync()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    torch.cuda._sleep(2_000_000_000)  # a second of other work on the default stream
    done = torch.cuda.Event()
    done.record()
    b.step(dt, ts, 2)
    waited = done.query()
    torch.cuda.synchronize()
    assert not waited
    b.close()
