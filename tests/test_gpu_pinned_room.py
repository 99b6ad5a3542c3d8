"""The pinned room through which a small grid's tables and fields cross: no context has
one before its second i2g_set_grid; with it, any fields given or left out, next to each
other or apart, give what a context that sets its grid once gives, bit for bit, and a
read-out of any node fields writes those and no others."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


def shared_megabytes():
    for line in open("/proc/self/status"):
        if line.startswith("RssShmem"):
            return int(line.split()[1]) / 1024
    pytest.skip("no RssShmem in /proc/self/status")


def test_contexts_that_set_their_grid_once_pin_no_room():
    inst = synth.make_instance("s", n=201, k=1, nsteps=1, seed=3)
    lib.MarkerStep.from_instance(inst).close()  # the runtime's own
    before = shared_megabytes()
    keep = [lib.MarkerStep.from_instance(inst) for _ in range(20)]
    held = shared_megabytes() - before
    for ms in keep:
        ms.close()
    assert held < 10, held  # twenty rooms are 72 MB


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [4, 90, 131, 201])  # 64 KB: eighteen fields at 21, one at 90
def test_fields_apart(n, precision):
    inst = synth.make_instance("g", n=n, k=2, nsteps=1, seed=9)
    r = np.random.default_rng(n)
    full = {k: 1e-14 * r.standard_normal(n * n) for k in ("exx", "eyy", "exy")}
    full.update({k: 1e6 * r.standard_normal(n * n) for k in ("sxx", "syy", "sxy")})
    full.update({k: inst.grid[k] for k in ("vx", "vy", "pr")}, mu=np.full(n * n, 1e19), ga=np.full(n * n, 0.1))
    sets = [("vx", "vy", "pr"), ("vx", "vy", "pr", "mu"), ("vy",), (), ("exx", "sxy", "mu", "vx", "vy"), tuple(full),
            ("vx", "vy", "pr", "eyy", "ga"), ("mu",)]
    ms = lib.MarkerStep.from_instance(inst, precision=precision)
    for names in sets:
        fields = {k: full[k] for k in names}
        once = lib.MarkerStep.from_instance(inst, precision=precision, upload=False)
        out = []
        for m in (ms, once):
            m.set_grid(inst.gx, inst.gy, **fields)
            m.set_nodes(**inst.nodes)
            m.set_markers(inst.x, inst.y, inst.T, inst.eta, inst.mtype)
            m.movemark(inst.timestep, inst.timesum, update_visc=True)
            m.ronurecalc(inst.timesum)
            out.append(dict(m.get_markers(), **m.get_nodes()))
        once.close()
        for k in out[0]:
            np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=f"{names} {k}")
    nodes = ms.get_nodes()
    for ask in (("tk",), ("ro", "po"), ("nd", "cp", "kt"), ("nu", "ht"), ()):
        got = {k: np.full(n * n, -7.0) for k in synth.NODE_OUT}
        ms._check(ms.lib.i2g_get_nodes(ms.h, *[abi.dptr(got[k]) if k in ask else None for k in synth.NODE_OUT]), "nodes")
        for k in synth.NODE_OUT:
            np.testing.assert_array_equal(got[k], nodes[k] if k in ask else np.full(n * n, -7.0), err_msg=f"{ask} {k}")
    ms.close()
