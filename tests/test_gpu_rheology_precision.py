"""The mixed form's viscosity update against the FP64 form where both read the same
inputs exactly (uniform pressure, strain rates and stresses that FP32 holds): the same
model in 64 bits, within the roundings of its products, quotients and powers.

The longest chain is the power law: some 12 operations of half a unit, exp and pow of
two units each, and the argument of pow enters its result times 1 / markmm <= 1: 16
units of 2^-53 cover it.  The Peierls iteration divides its error in s by up to
(1 - s / sig0) at each turn: 8 times that."""
import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu
UNIT = 2.0 ** -53


def dyadic(v):
    return float(np.float32(v))


@pytest.mark.parametrize("uniform", [True, False], ids=["uniform", "nonuniform"])
@pytest.mark.parametrize("law,units", [("power", 16), ("brittle", 16), ("peierls", 128)])
def test_viscosity_update_matches_fp64(law, units, uniform):
    inst = synth.make_instance("v", n=33, k=1, nsteps=1, seed=5)
    n = inst.marknum
    # cells of 2^14 (and 2^13) metres, the markers in their middles: weights of 1/2 and 0
    w = np.full(32, 2.0 ** 14)
    if not uniform:
        w[::2] = 2.0 ** 13
    inst.gx = inst.gy = np.concatenate([[0.0], np.cumsum(w)])
    inst.xsize = inst.ysize = inst.gx[-1]
    mid = 0.5 * (inst.gx[1:] + inst.gx[:-1])
    inst.x, inst.y = np.repeat(mid, 32), np.tile(mid, 32)
    inst.grid = {k: np.zeros(inst.nodenum) for k in inst.grid}
    inst.mtype[:] = 5
    inst.T[:] = 300.0 + 1400.0 * synth.rng_uniform(5, 1, n)
    inst.eta[:] = 10.0 ** (18 + 4 * synth.rng_uniform(5, 2, n))
    inst.grid["pr"][:] = dyadic(3e8)
    for k, v in (("exx", 2.0 ** -48), ("eyy", -2.0 ** -48), ("exy", 2.0 ** -47), ("sxx", 2.0 ** 24), ("syy", -2.0 ** 24),
                 ("sxy", 2.0 ** 25)):
        inst.grid[k][:] = v
    t = inst.types
    for k in ("marknu", "markdh", "markdv", "markss", "markmm", "markll", "marka0", "markb0", "marks0", "marks1"):
        t[k][5] = 0.0
    t["markn0"][5], t["markn1"][5] = 1e10, 1e40
    inst.scal["nubeg"], inst.scal["nuend"] = 1e10, 1e40
    if law == "power":
        t["marknu"][5], t["markdh"][5], t["markdv"][5], t["markss"][5], t["markmm"][5] = 1.97e17, 154000.0, 0.8, 1e4, 2.3
    elif law == "brittle":
        t["marknu"][5], t["markll"][5], t["marka0"][5], t["markb0"][5], t["marks1"][5] = 1e40, 0.6, 1e6, 0.4, 1e10
    else:
        t["marknu"][5], t["markdh"][5], t["marks0"][5], t["marks1"][5] = 1e40, 532000.0, 10.0 ** 7.8, 9.1e9
    out = []
    for precision in (abi.PREC_FP64, abi.PREC_MIXED):
        ms = lib.MarkerStep.from_instance(inst, precision=precision)
        ms.movemark(inst.timestep, inst.timesum, update_visc=True)
        out.append(ms.get_markers(fields=("x", "eta", "p")))
        ms.close()
    np.testing.assert_array_equal(out[0]["x"], out[1]["x"])
    want, got = out[0]["eta"], out[1]["eta"]
    assert np.unique(want).size > 100 and (want != inst.eta).all()
    err = np.abs(got / want - 1) / UNIT
    assert err.max() <= units, (err.max(), err.mean())
