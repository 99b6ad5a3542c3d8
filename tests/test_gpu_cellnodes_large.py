"""The one-lane-per-cell form of the fused averaging (grids of more than a CTA per SM)
where its buckets overflow and where nodes need quanta of their own, with the bars of
test_gpu_fused.py, whose cases of both are on a grid small enough for two lanes."""
import numpy as np
import pytest

from i2elvis_planet_b200 import synth
from test_gpu_batch_spill import gathering
from test_gpu_fused import check_against

pytestmark = pytest.mark.gpu
LINES = 187


@pytest.mark.parametrize("each", [5, 6, 43])  # 15, 18 and 129 records for buckets of 14, 14 and 64
def test_cells_beyond_their_buckets(each):
    mk, nodes, info = check_against(gathering(LINES, each, 8), nsteps=2)
    assert info["bucket_growths"] == 1, info


def test_sparse_nodes_take_the_guard():
    inst = synth.make_instance("c", n=LINES, k=2, nsteps=1, seed=12)
    n = LINES - 1
    m1, m2 = np.repeat(np.arange(n), n), np.tile(np.arange(n), n)
    u = synth.rng_uniform(4242, 1, n * n + 1000)
    w = synth.rng_uniform(4242, 2, 1000)
    dx = inst.gx[1] - inst.gx[0]
    sub = synth.subset(inst, np.arange(n * n + 1000))
    sub.x = np.concatenate([inst.gx[m1] + (1.0 - 1e-5 * (1 + u[:n * n])) * dx, inst.gx[90] + (0.05 + 0.9 * u[n * n:]) * dx])
    sub.y = np.concatenate([inst.gy[m2] + (1.0 - 1e-5 * (2 - u[:n * n])) * dx, inst.gy[101] + (0.05 + 0.9 * w) * dx])
    sub.grid = dict(inst.grid, vx=np.zeros_like(inst.grid["vx"]), vy=np.zeros_like(inst.grid["vy"]))
    check_against(sub, nsteps=1)
