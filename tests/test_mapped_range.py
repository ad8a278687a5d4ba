"""Which host arrays a run reads and writes in place (cans::mapped_range), with made-up
registrations: an array whose ends lie in two registrations but whose middle is in none
is not page-locked.  CPU only; no memory is touched."""
import ctypes as C

import pytest

from utrip_gb300 import build

PAGE = 4096
BASE = 1 << 40


@pytest.fixture(scope="module")
def mapped():
    build.build()
    lib = C.CDLL(str(build.LIBDIR / build.PROBELIB))
    u = C.c_ulonglong
    lib.cans_probe_mapped_range.argtypes = [u, u, u, C.POINTER(u), C.POINTER(u), C.c_int]

    def ask(start, n, segs, shifts=None):
        """An array of n doubles from byte `start`; segs in pages [lo, hi)."""
        flat = [BASE + PAGE * e for s in segs for e in s]
        shifts = [0] * len(segs) if shifts is None else shifts
        return bool(lib.cans_probe_mapped_range(BASE + start, n, PAGE, (u * len(flat))(*flat),
                                                (u * len(segs))(*shifts), len(segs)))
    return ask


@pytest.mark.parametrize("start", [0, 8, 4088, 4096, 5000 * 8])
@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 1026, 5000])
def test_whole_registrations_pass(mapped, start, n):
    lo, hi = start // PAGE, (start + 8 * n - 1) // PAGE + 1
    assert mapped(start, n, [(lo, hi)])
    assert mapped(start, n, [(lo, hi)], [1 << 30])
    if hi - lo > 1:
        assert mapped(start, n, [(lo, lo + 1), (lo + 1, hi)])  # side by side
        assert not mapped(start, n, [(lo + 1, hi)])
        assert not mapped(start, n, [(lo, hi - 1)])
        assert not mapped(start, n, [(lo, lo + 1), (lo + 1, hi)], [0, PAGE])
    assert not mapped(start, n, [])


@pytest.mark.parametrize("start", [0, 8, 4088])
@pytest.mark.parametrize("n", [1026, 5000])
def test_a_hole_between_two_registrations_is_seen(mapped, start, n):
    pages = (start + 8 * n - 1) // PAGE + 1
    for lo in range(1, pages - 1):
        assert not mapped(start, n, [(0, lo), (lo + 1, pages)]), lo


def test_misaligned_and_empty(mapped):
    assert not mapped(4, 10, [(0, 1)])
    assert not mapped(0, 0, [(0, 1)])
