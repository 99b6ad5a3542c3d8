"""Rounding of the fused averaging's cell sums and means, on records whose exact sums
are known: n equal markers in one cell of a grid that does not move.

Every term of a sum is rounded to a multiple of u, half the spacing of doubles at the
sum's start (2^(e-53), 2^e the power of two above 4 max(n, 4) (1 + 2^-20) times the
largest term), to the nearest: a sum of n terms is off by n u / 2 at most, where
rounding down would cost these records 3/4 u each.  A mean is the correctly rounded
quotient of its two sums."""
import math

import numpy as np
import pytest

from i2elvis_planet_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu
UNIT = 2.0 ** -53


def crowd(n, lines, a, b, T, eta, viscmod=1):
    """n markers with T and eta at x = a 2^-23, y = b 2^-23 (from -1 to 1 across a cell)
    of the cell at the box's centre."""
    inst = synth.make_instance("r", n=lines, k=1, nsteps=1, seed=3)
    inst = synth.subset(inst, np.arange(n))
    w = inst.xsize / (lines - 1)
    c = (lines - 1) // 2
    inst.x[:] = (c + (2 ** 23 + a) / 2 ** 24) * w
    inst.y[:] = (c + (2 ** 23 + b) / 2 ** 24) * w
    inst.T[:], inst.eta[:], inst.mtype[:] = T, eta, 5
    inst.flags["viscmod"] = viscmod
    inst.grid = {k: np.zeros(inst.nodenum) for k in inst.grid}
    ms = lib.MarkerStep.from_instance(inst, precision=abi.PREC_MIXED)
    ms.movemark(inst.timestep, inst.timesum)
    ms.ronurecalc(inst.timesum)
    assert ms.fused_info()["fused_moves"] == 1
    nodes = {k: v.reshape(lines, lines) for k, v in ms.get_nodes().items()}
    ms.close()
    return inst, nodes, c


def unit(n, largest):
    return 2.0 ** (math.floor(math.log2(4 * max(n, 4) * (1 + 2.0 ** -20) * largest)) + 1 - 53)


@pytest.mark.parametrize("lines", [33, 193], ids=["two-lanes", "one-lane"])
@pytest.mark.parametrize("n", [77, 160, 161])  # u = 4 and more times the last bit of T x
def test_temperature_terms_round_to_nearest(lines, n):
    m = 700 * 2 ** 14 + 1  # T = m 2^-14
    a = -pow(m, -1, 2 ** 22) % 2 ** 22  # x = a 2^-23: T x = -2^-37 modulo 2^-15
    T = m * 2.0 ** -14
    inst, nodes, c = crowd(n, lines, a, 0, T, 1e19)
    u = unit(n, T)
    assert 2.0 ** -37 < u < 2.0 ** -30
    x = a * 2.0 ** -23
    for p in (0, 1):
        # the mean of equal temperatures: off by the sum's n u / 2 against n T (1 -+ x), and two roundings
        bound = 0.5 * u / (T * (1 + x if p else 1 - x)) + 2 * UNIT
        for q in (0, 1):
            got = nodes["tk"][c + p, c + q]
            assert abs(got / T - 1) <= bound, (p, q, (got / T - 1) / bound)


@pytest.mark.parametrize("lines", [33, 193], ids=["two-lanes", "one-lane"])
@pytest.mark.parametrize("n", [40, 77])
def test_cell_centre_viscosity_rounds_to_nearest(lines, n):
    """viscmod 0: the cell-centre viscosity is the mean of equal viscosities with the
    tent weight c = (1 - |x|)(1 - |y|), here a multiple of its sum's u: the sum of the
    weights is exact, that of the products is off by n u / 2."""
    eta = 3456789013 * 2.0 ** 35  # 32 significant bits: as the record holds it
    uw, un = unit(n, 1.0), unit(n, eta)
    b = 2 ** 22

    bits = 11 + round(math.log2(un))  # eta c = 3456789013 (2^23 - a) (2^23 - b) 2^-11
    a = next(k for k in range(2 ** 21, 2 ** 22, 8)
             if 0.9 < 3456789013 * (2 ** 23 - k) * (2 ** 23 - b) % 2 ** bits / 2 ** bits < 0.99)
    w = (1 - a * 2.0 ** -23) * (1 - b * 2.0 ** -23)
    assert w % uw == 0
    inst, nodes, c = crowd(n, lines, a, b, 512.0, eta, viscmod=0)
    bound = 0.5 * un / (eta * w) + 2 * UNIT
    got = nodes["nd"][c + 1, c + 1]
    assert abs(got / eta - 1) <= bound, (got / eta - 1) / bound


@pytest.mark.parametrize("lines", [33, 193], ids=["two-lanes", "one-lane"])
def test_means_are_quotients(lines):
    """49 markers in the middle of a cell: every weight sum is 49/4, and a product with
    it divides back to the value (times its reciprocal it does not)."""
    for cp, kt in ((1000.0, 3.0), (800.0, 40.0)):
        inst, nodes, c = crowd(49, lines, 0, 0, 512.0, 1e19)
        t = inst.types
        assert (t["markcp"][5] * 12.25) * (1 / 12.25) != t["markcp"][5]
        at = np.s_[c:c + 2, c:c + 2]
        np.testing.assert_array_equal(nodes["ro"][at], t["markro"][5])
        np.testing.assert_array_equal(nodes["cp"][at], t["markcp"][5])
        np.testing.assert_array_equal(nodes["kt"][at], t["markkt"][5])
