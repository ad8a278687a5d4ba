"""The integer-pipe sums of csrc/isum.cuh against exactly rounded sums
(math.fsum): operands within 2^7 of the largest enter exactly, so their sum is
the nearest double; a smaller operand is truncated below 2^-60 of the largest,
so four of them leave the sum within 2^-58 of it before its rounding."""
import ctypes as C
import math
from fractions import Fraction

import numpy as np
import pytest

from utrip_gb300 import build

pytestmark = pytest.mark.gpu


def sums(x):
    lib = C.CDLL(str(build.LIBDIR / build.PROBELIB))
    x = np.ascontiguousarray(x, dtype=np.float64)
    n = len(x)
    y, f = np.empty((n, 2)), np.empty(n, dtype=np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert lib.cans_probe_isum(p(x), p(y), p(f), C.c_int(n)) == 0
    return y, f != 0


def exact(x):
    return np.array([[math.fsum(r), math.fsum((r[1], -r[0], r[2], -r[3]))] for r in x])


def operands(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    x = np.ldexp(rng.uniform(0.5, 1.0, (n, 4)), rng.integers(lo, hi + 1, (n, 4)))
    return x * rng.choice([-1.0, 1.0], (n, 4))


@pytest.mark.parametrize("shift", [-900, -30, 0, 1, 500, 1010])
def test_near_operands_are_rounded_once(shift):
    x = np.concatenate([operands(20000, 0, 6, 1), operands(20000, 0, 0, 2),
                        np.round(operands(20000, 3, 3, 3)),       # exact sums, many ties
                        np.repeat(operands(500, 0, 0, 4)[:, :1], 4, axis=1)])  # cancel to zero
    x[::7, 2] = 0.0
    x[::11, 0] = -0.0
    x[::13] = np.nextafter(x[::13], 0.0)
    x = np.ldexp(x, shift)
    y, sp = sums(x)
    assert not sp.any()
    assert np.array_equal(y, exact(x))


def test_wide_operands():
    x = operands(60000, -80, 0, 5)
    y, sp = sums(x)
    assert not sp.any()
    big = np.max(np.abs(x), axis=1)
    for r, got, m in zip(x, y, big):  # against the sums unrounded
        a, b, c, d = (Fraction(v) for v in r)
        for g, want in zip(got, (a + b + c + d, (b - a) + (c - d))):
            err = float(abs(Fraction(g) - want))
            assert err <= 2.0 ** -58 * m + 0.5000001 * np.spacing(abs(g)), (r, g)


def test_zeros_and_what_is_left_to_fp64():
    tiny = 5e-324
    x = np.array([[0.0, -0.0, 0.0, 0.0], [1.0, 0.0, 0.0, 0.0], [tiny, 0, 0, 0],
                  [0, 0, 0, 1e-310], [2.0 ** -960, 0, 0, 0], [1e-300, -1e-300, 0, 0],
                  [np.inf, 0, 0, 0], [0, np.nan, 1, 1], [1.7e308, 1, 1, 1],
                  [1.0, tiny, -tiny, 0.0]])
    y, sp = sums(x)
    assert list(sp) == [False, False, True, True, True, True, True, True, True, False]
    assert np.array_equal(y[[0, 1, 9]], [[0, 0], [1, -1], [1, -1]])
