"""The two-operand additions of csrc/isum.cuh and the minmod face states formed with
them against FP64: the same bits (no tolerance), for near, wide, cancelling and tied
operands and zeros; operands beyond the range are flagged, and the face states
take FP64 there."""
import ctypes as C

import numpy as np
import pytest
import torch

from utrip_gb300 import build

pytestmark = pytest.mark.gpu


def lib():
    return C.CDLL(str(build.LIBDIR / build.PROBELIB))


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def add2(x, y):
    x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
    z, f = np.empty(len(x)), np.empty(len(x), dtype=np.int32)
    assert lib().cans_probe_add2(ptr(x), ptr(y), ptr(z), ptr(f), C.c_int(len(x))) == 0
    return z, f != 0


def draw(n, spread, seed):
    rng = np.random.default_rng(seed)
    m = np.where(rng.random(n) < 0.5, rng.uniform(1.0, 2.0, n),
                 1.0 + rng.integers(0, 8, n) * 2.0 ** -rng.integers(1, 53, n))  # few bits: ties
    return np.ldexp(m, rng.integers(-spread, spread + 1, n)) * rng.choice([-1.0, 1.0], n)


@pytest.mark.parametrize("spread", [0, 1, 2, 12, 40, 80, 400])
def test_add2_is_the_fp64_sum(spread):
    n = 200000
    x, y = draw(n, spread, 1), draw(n, spread, 2)
    y[::5] = -np.nextafter(x[::5], 2.0)            # cancel to the last bits
    y[1::11] = -x[1::11]                           # to zero
    y[2::11] = x[2::11] * 2.0 ** -53               # a half of the last place
    y[3::11] = -x[3::11] * 2.0 ** -54
    x[4::13], y[5::13] = 0.0, -0.0
    x[6::26], y[6::26] = -0.0, -0.0
    z, sp = add2(x, y)
    assert not sp.any()
    assert np.array_equal(z.view(np.int64), (x + y).view(np.int64))


def test_add2_flags_what_it_cannot_form():
    x = np.array([5e-324, 1e-310, 1e-300, np.inf, -np.inf, np.nan, 1.7e308, 0.0, 5e-324])
    y = np.array([0.0, 1.0, 1e-300, 1.0, np.inf, 1.0, 1.7e308, np.nan, -5e-324])
    z, sp = add2(x, y)
    assert list(sp) == [True, False, True, True, True, True, True, True, True]
    assert z[1] == 1.0


@pytest.mark.parametrize("spread", [0, 3, 60])
@pytest.mark.parametrize("scale", [0, -900, 962])
def test_face_states_are_those_of_fp64(scale, spread):
    n = 100000
    x = np.ldexp(np.stack([draw(n, spread, 3 + k) for k in range(4)], axis=1), scale)
    x[::3] = np.sort(x[::3], axis=1)               # monotone: minmod is not zero
    x[1::7, 1] = x[1::7, 0]
    x[2::9] = 0.0
    x = np.ascontiguousarray(x)
    y = np.empty((n, 2))
    assert lib().cans_probe_muscl(ptr(x), ptr(y), C.c_int(n)) == 0
    # FP64 on the device, as the sign of inf - inf is the device's
    dm, d0, d1, d2 = torch.from_numpy(x.T.copy()).cuda()

    def minmod(a, b):
        # the smaller magnitude by bit pattern, as the kernels compare: a NaN is beyond inf
        p, q = (v.view(torch.int64) & (2 ** 63 - 1) for v in (a, b))
        m = torch.minimum(p, q).view(torch.float64)
        a_neg, b_neg = a.view(torch.int64) < 0, b.view(torch.int64) < 0
        return torch.where(a_neg == b_neg, torch.where(a_neg, -m, m), torch.zeros_like(m))

    # one rounding each, as m / 2 is exact (no subnormal differences)
    want = torch.stack([d0 + 0.5 * minmod(d0 - dm, d1 - d0), d1 - 0.5 * minmod(d2 - d1, d1 - d0)],
                       dim=1).cpu().numpy()
    assert np.array_equal(y, want, equal_nan=True)
