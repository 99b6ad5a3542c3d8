"""Identities the device code relies on, checked against the host C library the
reference links (no GPU needed).

The viscosity update evaluates the reference's pow(v, 0.5) (strain-rate and stress
invariants, markmart.c:47-48; the Peierls iteration of viscalc, markmart.c:1923)
as sqrt(v), with pow's results for -0 (+0) and -inf (+inf).  glibc's pow is not
correctly rounded, so for a small fraction of doubles the two differ by one unit
in the last place; never by more, and never in the special values."""
import ctypes as C
import ctypes.util
import os
import re

import numpy as np

libm = C.CDLL(ctypes.util.find_library("m"))
libm.pow.restype = C.c_double
libm.pow.argtypes = [C.c_double, C.c_double]
libm.sqrt.restype = C.c_double
libm.sqrt.argtypes = [C.c_double]


def pow_half(v: float) -> float:
    """The device's evaluation (i2g_dev.cuh: pow_half)."""
    return float("inf") if v == float("-inf") else libm.sqrt(v) + 0.0


def ulps(a: float, b: float) -> int:
    if np.isnan(a) and np.isnan(b):
        return 0
    ia, ib = np.float64(a).view(np.int64), np.float64(b).view(np.int64)
    return abs(int(ia) - int(ib))


def test_sqrt_within_one_ulp_of_pow_half():
    rng = np.random.default_rng(20261203)
    values = np.concatenate([
        rng.random(20000) * 10.0 ** rng.integers(-300, 300, 20000),   # positive normals
        np.frombuffer(rng.integers(1, 2 ** 52, 2000, dtype=np.uint64).tobytes(), dtype=np.float64),  # subnormals
        -rng.random(200),                                            # negatives: NaN from both
        np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1.7976931348623157e308, 1.0, 4.0]),
    ])
    diff = np.array([ulps(pow_half(float(v)), libm.pow(float(v), 0.5)) for v in values])
    assert diff.max() <= 1
    assert (diff > 0).mean() < 0.01
    for v in (0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, 1.0, 4.0, 5e-324):
        assert ulps(pow_half(v), libm.pow(v, 0.5)) == 0, v
        assert np.signbit(pow_half(v)) == np.signbit(libm.pow(v, 0.5)) or np.isnan(v) or v < 0, v


def test_div_by_is_the_division():
    """div_by (i2g_dev.cuh): a / h from r = 1 / h by two corrections, every result
    the IEEE quotient: random numerators, and ones whose quotient lies next to a
    double or halfway between two, for widths of grids and extreme ones."""
    libm.fma.restype = C.c_double
    libm.fma.argtypes = [C.c_double] * 3
    rng = np.random.default_rng(7)
    n = 40000
    h = np.concatenate([rng.random(n) * 10.0 ** rng.integers(-3, 7, n), 500.0 * (1 + 2.0 ** -52 * rng.integers(0, 4000, n)),
                        np.ldexp(1 + rng.random(n), rng.integers(-390, 390, n)), np.full(n, 6.0)])
    q = rng.random(h.size)
    half = np.nextafter(q, 1) * 0.5 + q * 0.5
    with np.errstate(under="ignore"):
        a = np.where(rng.random(h.size) < 0.3, q * h, np.where(rng.random(h.size) < 0.5, half * h, rng.random(h.size) * h))
        a = np.where(rng.random(h.size) < 0.5, a, np.nextafter(a, np.where(rng.random(h.size) < 0.5, np.inf, -np.inf)))
    a = a * np.where(rng.random(h.size) < 0.5, 1.0, -1.0)
    a = a[np.abs(a) >= 2.0 ** -900][: h.size]
    h = h[: a.size]
    bad = 0
    for x, w in zip(a.tolist(), h.tolist()):
        r = 1.0 / w
        v = x * r
        v = libm.fma(libm.fma(-v, w, x), r, v)
        v = libm.fma(libm.fma(-v, w, x), r, v)
        bad += v != x / w
    assert bad == 0


def test_div_by_at_the_ends_of_its_range():
    """div_by where the device code still uses it: numerators down to kDivTiny
    (i2g_dev.cuh) against the narrowest and widest cells that fill_axis (i2g_api.cu)
    takes into its tables; no product underflows there."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "i2elvis_planet_b200", "csrc")
    tiny = int(re.search(r"kDivTiny = \(1023u - (\d+)u\)", open(os.path.join(csrc, "i2g_dev.cuh")).read()).group(1))
    low, high = map(int, re.search(r"h > 0x1p-(\d+) && h < 0x1p(\d+)", open(os.path.join(csrc, "i2g_api.cu")).read()).groups())
    libm.fma.restype = C.c_double
    libm.fma.argtypes = [C.c_double] * 3
    rng = np.random.default_rng(8)
    n = 20000
    h = np.ldexp(1 + rng.random(n), rng.integers(-low, high, n))
    a = np.ldexp(1 + rng.random(n), rng.integers(-tiny, 60 - tiny, n)) * np.where(rng.random(n) < 0.5, 1.0, -1.0)
    # and, where widths reach that far, quotients halfway between two subnormals
    h[::2] = np.ldexp(1 + rng.integers(0, 2 ** 20, h[::2].size) / 2.0 ** 20, rng.integers(-low, high, h[::2].size))
    half = np.ldexp(h * (2 * rng.integers(1, 2 ** 30, n) + 1), -1075)
    a[::2] = np.where((half >= 2.0 ** -tiny)[::2], half[::2], a[::2])
    bad = 0
    for x, w in zip(a.tolist(), h.tolist()):
        r = 1.0 / w
        v = x * r
        v = libm.fma(libm.fma(-v, w, x), r, v)
        v = libm.fma(libm.fma(-v, w, x), r, v)
        bad += v != x / w
    assert bad == 0
