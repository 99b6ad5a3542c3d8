"""The fused averaging's cell sums at the edges of its tiles and shapes: grids around
multiples of 31 and 15 node rows and on both sides of the two-lanes-per-cell rule,
one to four type slots (one of them immobile), cells with no, one, two, odd and
many records.

Oracle: the records as the step forms them, weights rounded to 24 bits and T to FP32
at the positions the context reports, summed in numpy FP64.  Bars: the sums keep
weights and means each within 1e-9 (the rounding quanta's bound), so 2e-9 for the
fields made of weights and temperature; a node viscosity adds the mixed form's
logarithm, log2f of an FP32 mantissa: 1.5e-7 at most.  Another order of the markers
gives the same bits."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


def instance(n, per_cell, types, immobile):
    inst = synth.make_instance("e", n=n, k=max(1, int(np.ceil(np.sqrt(per_cell)))), nsteps=1, seed=11)
    u = synth.rng_uniform(77, n, inst.marknum)
    keep = np.nonzero(u < per_cell / inst.mnumx ** 2)[0]
    inst = synth.subset(inst, keep if keep.size else np.arange(1))
    pick = (synth.rng_uniform(78, n, inst.marknum) * len(types)).astype(int)
    inst.mtype = np.array(types, dtype=np.int8)[pick]
    for t in types:
        inst.types["markro"][t] = 1000.0 + 100.0 * t
        inst.types["markcp"][t] = 900.0 + 10.0 * t
    if immobile:
        inst.markim[types[-1]] = 1
    inst.nodes["tk"][:] = 321.0
    return inst


def run(inst):
    ms = lib.MarkerStep.from_instance(inst, precision=abi.PREC_MIXED)
    ms.step(inst.timestep, inst.timesum, 2)
    out = ms.get_nodes(), ms.get_markers(), ms.fused_info(), ms.stats().markers_averaged
    ms.close()
    return out


def weights(g, v):
    """Cell and upper weight on a uniform axis, the weight to 24 bits (round to even)."""
    w = (g[-1] - g[0]) / (g.size - 1)
    b = np.clip(np.floor((v - g[0]) * (1.0 / w)).astype(np.int64), 0, g.size - 2)
    line = (b.astype(np.longdouble) * np.longdouble(w) + np.longdouble(g[0])).astype(np.float64)  # one rounding
    return b, np.rint(np.clip((v - line) * (1.0 / w), 0.0, 1.0) * 2.0 ** 24) / 2.0 ** 24


def expected(inst, mk):
    x, y, T = mk["x"], mk["y"], mk["T"]
    L = inst.xsize
    ok = (x > 0) & (y > 0) & (x < L) & (y < L) & (T > 0)
    t = inst.mtype.astype(int)[ok]
    x, y = x[ok], y[ok]
    T = np.where(t < 2, inst.scal["tmp_ambient"], T[ok]).astype(np.float32).astype(np.float64)
    eta = np.where(np.hypot(x - L / 2, y - L / 2) > 0.95 * L / 2, 1e22, mk["eta"][ok])
    a, X = weights(inst.gx, x)
    b, Y = weights(inst.gy, y)
    ny, nn = inst.ynumy, inst.nodenum
    out = {k: np.zeros(nn) for k in ("w", "w1", "tk", "ro", "cp", "wnu", "nu", "wnd", "nd")}
    mobile = inst.markim[t] == 0
    for p in (0, 1):
        for q in (0, 1):
            i = (a + p) * ny + b + q
            wx, wy = (X if p else 1 - X), (Y if q else 1 - Y)
            w = wx * wy
            for k, v in (("w", w), ("w1", w * mobile), ("tk", w * mobile * T), ("ro", w * inst.types["markro"][t]),
                         ("cp", w * inst.types["markcp"][t])):
                np.add.at(out[k], i, v)
            s = np.where((wx > 0.5) & (wy > 0.5), 4 * (wx - 0.5) * (wy - 0.5), 0.0)
            np.add.at(out["wnu"], i, s)
            np.add.at(out["nu"], i, s * np.log(eta))
    s = 4 * (0.5 - np.abs(X - 0.5)) * (0.5 - np.abs(Y - 0.5))
    np.add.at(out["wnd"], (a + 1) * ny + b + 1, s)
    np.add.at(out["nd"], (a + 1) * ny + b + 1, s * np.log(eta))
    return out, int(ok.sum())


@pytest.mark.parametrize("n,per_cell,types,immobile", [
    (3, 1.0, (5,), False), (16, 3.0, (0, 5), False), (17, 0.4, (0, 5, 7), False), (31, 2.5, (0, 5, 7, 8), True),
    (32, 7.0, (5, 7, 8), True), (33, 16.0, (0, 5, 7), False), (63, 1.3, (0, 5, 7, 8), False), (64, 9.0, (5, 7), True),
    (105, 5.0, (0, 5, 7), False), (121, 3.3, (0, 5, 7, 9), True), (156, 2.0, (5,), False), (187, 11.0, (0, 5, 7), False),
])
def test_cell_sums_at_edges(n, per_cell, types, immobile):
    inst = instance(n, per_cell, types, immobile)
    nodes, mk, info, averaged = run(inst)
    assert info["fused_moves"] == 2
    want, count = expected(inst, mk)
    assert averaged == count
    with np.errstate(divide="ignore", invalid="ignore"):
        for k, w, tol in (("ro", "w", 2e-9), ("cp", "w", 2e-9), ("tk", "w1", 2e-9), ("nu", "wnu", 1.6e-7), ("nd", "wnd", 1.6e-7)):
            v = want[k] / want[w]
            v = np.clip(np.exp(v), inst.scal["nubeg"], inst.scal["nuend"]) if k in ("nu", "nd") else v
            at = want[w] > 0
            assert np.abs(nodes[k][at] / v[at] - 1).max() <= tol, (k, np.abs(nodes[k][at] / v[at] - 1).max())
    perm = np.argsort(synth.rng_u64(9, n, inst.marknum), kind="stable")
    other = run(synth.subset(inst, perm))[0]
    for k in synth.NODE_OUT:
        np.testing.assert_array_equal(other[k], nodes[k], err_msg=k)
