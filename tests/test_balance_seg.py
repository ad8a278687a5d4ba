"""The rows of a segment of the marching 2-D steps (cans::balance_seg): the cheapest of
every length under its cost model, the shortest of equals, found without trying every
length (the launch of every drop-in step searches).  CPU only."""
import ctypes as C
import time

import pytest

from utrip_gb300 import build


@pytest.fixture(scope="module")
def probe():
    build.build()
    return C.CDLL(str(build.LIBDIR / build.PROBELIB))


def cheapest(strips, rows, ch, sms):
    def cost(seg):
        per_sm = -(-strips * -(-rows // seg) // sms)
        chunks = -(-seg // ch)
        return (per_sm // 2 * (80 + 40 * chunks + 18 * seg) +
                per_sm % 2 * (75 + 25 * chunks + 11 * seg))
    return min(range(1, rows + 1), key=cost)  # the first of equals


@pytest.mark.parametrize("ch", [6, 7, 8])
@pytest.mark.parametrize("strips", [1, 2, 7, 16, 64, 300])
def test_the_cheapest_segment(probe, strips, ch):
    for rows in [*range(1, 40), 63, 64, 126, 254, 255, 382, 510, 1022, 2046]:
        assert probe.cans_probe_balance_seg(strips, rows, ch, 152) == \
            cheapest(strips, rows, ch, 152), rows


def test_the_search_is_short(probe):
    """200 searches over 400000 rows: some 250000 candidates, where every length would
    be 80 million (half a second)."""
    t = time.perf_counter()
    for _ in range(200):
        probe.cans_probe_balance_seg(12500, 400000, 7, 152)
    assert time.perf_counter() - t < 0.1
