"""The FP64 reciprocals, roots and comparisons of csrc/fd64.cuh against extended
precision, over their whole range and at the edges of their seeds.

The bounds are those of the Newton step: rcp and sqrt add a rounded
correction to a seed whose error, squared, is below 2^-90 (0.51 ulp); rsqrt
rounds x y once before the correction (1 ulp)."""
import ctypes as C

import numpy as np
import pytest

from utrip_gb300 import build

pytestmark = pytest.mark.gpu
_dp = C.POINTER(C.c_double)


def probe(op, x, w=None):
    lib = C.CDLL(str(build.LIBDIR / build.PROBELIB))
    lib.cans_probe_fd64.argtypes = [C.c_int, _dp, _dp, _dp, C.c_int]
    x = np.ascontiguousarray(x, dtype=np.float64)
    w = x if w is None else np.ascontiguousarray(w, dtype=np.float64)
    y = np.empty_like(x)
    assert lib.cans_probe_fd64(op, *[a.ctypes.data_as(_dp) for a in (x, w, y)], x.size) == 0
    return y


def arguments(seed):
    rng = np.random.default_rng(seed)
    m = 1.0 + rng.random(400000)
    wide = np.ldexp(m, rng.integers(-1019, 1020, m.size))
    near = np.ldexp(m, rng.integers(-2, 3, m.size))
    one = np.array([1.0, 2.0, 4.0, 0.5, 0.25])
    edges = np.concatenate([one, np.nextafter(one, 8), np.nextafter(one, 0),
                            one * (1 + 2.0 ** -24), one * (1 - 2.0 ** -25),
                            one * (1 + 2.0 ** -23 - 2.0 ** -52)])
    head = np.float64(np.float32(near[:100000]))  # no rest below the float
    return np.concatenate([wide, near, edges, head, np.nextafter(head, 0),
                           np.nextafter(head, 8)])


def ulps(got, want):
    want = want.astype(np.longdouble)
    return np.max(np.abs(got.astype(np.longdouble) - want) /
                  np.spacing(np.abs(want).astype(np.float64)).astype(np.longdouble))


@pytest.mark.parametrize("op,bound", [(0, 0.51), (1, 0.51), (2, 1.0), (3, 0.51), (4, 1.0)])
def test_error(op, bound):
    x = arguments(op)
    e = x.astype(np.longdouble)
    want = {0: 1 / e, 1: np.sqrt(e), 2: 1 / np.sqrt(e), 3: np.sqrt(e), 4: 1 / np.sqrt(e)}[op]
    assert ulps(probe(op, x), want) <= bound
    if op == 0:
        assert np.array_equal(probe(0, -x), -probe(0, x))


def test_special_arguments():
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, 2.2250738585072014e-308,
                  4.4e-308, 1.7e308, 4.4e307, -1.0])
    with np.errstate(all="ignore"):
        for op, want in ((0, 1.0 / x), (1, np.sqrt(x)), (3, np.sqrt(x))):
            got = probe(op, x)
            ok = np.isfinite(want) & (want != 0)
            assert np.array_equal(got[~ok], want[~ok], equal_nan=True), op
            assert np.all(np.abs(got[ok] - want[ok]) <= np.spacing(np.abs(want[ok]))), op
        assert np.array_equal(np.isnan(probe(2, x)), np.isnan(1.0 / np.sqrt(x)))


def test_comparisons():
    v = np.array([-np.inf, -1e300, -2.0, -1.0 - 2 ** -52, -1.0, -1e-310, 0.0, 5e-324, 1e-10,
                  1.0, 1.0 + 2 ** -52, 3e300, np.inf])
    a, b = (q.reshape(-1) for q in np.meshgrid(v, v))
    assert np.array_equal(probe(5, a, b), (a < b).astype(float))
    assert np.array_equal(probe(6, a, b), np.maximum(a, b))
    assert np.array_equal(probe(7, v), np.maximum(v, 0.0))
