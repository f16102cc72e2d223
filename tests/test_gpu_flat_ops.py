"""gb::FlatOps (flat_ops.cuh), the quotients and roots without branches: the
IEEE results wherever they say that their operands are in range, except that a
quotient within 2^-52 ulp of the midpoint of two doubles may take the farther
one and a numerator below 2^-960 is held to an ulp (or 2^-1074); and out of
range everywhere else (the caller then uses the plain operators)."""
import ctypes
import os
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gamma_b200", "lib",
                   "libgamma_selftest.so")
QUO, INV, ROOT, RROOT = 1, 2, 4, 8


def _flat(a, b):
    lib = ctypes.CDLL(LIB)
    p = lambda v, t: v.ctypes.data_as(ctypes.POINTER(t))  # noqa: E731
    out, bad = np.zeros((4, a.size)), np.zeros(a.size, np.int32)
    assert lib.gb_selftest_flat_ops(p(a, ctypes.c_double), p(b, ctypes.c_double), p(out, ctypes.c_double),
                                    p(bad, ctypes.c_int), a.size) == 0
    return out, bad


def _pairs(kind):
    rng = np.random.default_rng(11)
    n = 400000
    m = lambda: 1. + rng.integers(0, 2 ** 52, n) * 2. ** -52  # noqa: E731  significands
    if kind == "random":
        return m() * rng.choice([-1., 1.], n) * 2. ** rng.integers(-440, 440, n), m() * 2. ** rng.integers(-440, 440, n)
    if kind == "near_one":  # 1 +- k ulp: exact powers, significands of all ones, ties of the root
        k = rng.integers(-6, 7, n) * 2. ** -53
        j = rng.integers(-6, 7, n) * 2. ** -53
        e = 2. ** rng.integers(-3, 4, n)
        return (1. + k) * e, (1. + j) * 2. ** rng.integers(-3, 4, n)
    if kind == "all_ones":
        return m() * 2. ** rng.integers(-20, 20, n), (2. - 2. ** -52) * 2. ** rng.integers(-20, 20, n)
    if kind == "midpoints":  # a = RN(b (q + ulp/2)): quotients next to a midpoint; a = RN(q^2): roots
        b, q = m(), m()
        half = q + 2. ** -53 * 0.
        hi = b * half
        return np.where(np.arange(n) % 2 == 0, hi + b * 2. ** -53, half * half + half * 2. ** -52), b
    if kind == "tiny":  # numerators down to the smallest subnormals
        return m() * 2. ** rng.integers(-1074, -700, n).astype(float), m() * 2. ** rng.integers(-60, 60, n)
    if kind == "zeros":
        a = np.where(rng.random(n) < .5, 0., -0.)
        return a, m() * rng.choice([-1., 1.], n) * 2. ** rng.integers(-440, 440, n)
    special = np.array([0., -0., 5e-324, -5e-324, 1e-310, 2.0 ** -600, 2.0 ** -451, 2.0 ** -450, 2.0 ** 450,
                        2.0 ** 452, 1e200, np.inf, -np.inf, np.nan, 1., -1.])
    return np.repeat(special, special.size), np.tile(special, special.size)


def _tie(a, b, got, want):
    """Whether a/b lies within 2^-51 ulp of the midpoint of got and want, neighbours."""
    g, w = Fraction(float(got)), Fraction(float(want))
    ulp = Fraction(float(np.spacing(abs(want))))
    return abs(g - w) <= ulp and abs(Fraction(float(a)) / Fraction(float(b)) - (g + w) / 2) <= ulp / 2 ** 51


@pytest.mark.parametrize("kind", ["random", "near_one", "all_ones", "midpoints", "zeros", "tiny", "special"])
def test_flat_ops_are_ieee_in_range(gpu_available, kind):
    a, b = (np.ascontiguousarray(v, dtype=np.float64) for v in _pairs(kind))
    out, bad = _flat(a, b)
    with np.errstate(all="ignore"):
        want = np.stack([a / b, 1. / b, np.sqrt(a), 1. / np.sqrt(a)])
    for k, bit in enumerate((QUO, INV, ROOT, RROOT)):
        ok = (bad & bit) == 0
        same = (out[k].view(np.uint64) == want[k].view(np.uint64)) | (np.isnan(out[k]) & np.isnan(want[k]))
        if bit == QUO:
            with np.errstate(all="ignore"):
                same |= (np.abs(a) < 2. ** -960) & (np.abs(out[k] - want[k]) <= np.spacing(np.abs(want[k])))
        wrong = np.flatnonzero(ok & ~same)
        if bit == QUO:
            wrong = np.array([i for i in wrong if not _tie(a[i], b[i], out[k][i], want[k][i])], dtype=int)
        assert wrong.size == 0, (kind, bit, a[wrong[:4]], b[wrong[:4]], out[k][wrong[:4]], want[k][wrong[:4]])
        if kind not in ("special", "tiny"):
            assert ok.all() or (kind == "zeros" and bit == RROOT)
    if kind == "tiny":
        assert ((bad & QUO) == 0).all()
    if kind == "special":  # what must not pass as in range
        big = lambda v: ~np.isfinite(v) | (np.abs(v) > 2. ** 451)  # noqa: E731
        out_of = lambda v: big(v) | (np.abs(v) < 2. ** -450)  # noqa: E731
        assert ((bad & QUO) != 0)[big(a) | out_of(b)].all()
        assert ((bad & INV) != 0)[out_of(b)].all()
        assert ((bad & ROOT) != 0)[out_of(a) & (a != 0.)].all()
        assert ((bad & RROOT) != 0)[out_of(a)].all()
