"""When the rules of a 2-D boundary program may be applied in one pass over the frame
(cans::bc_one_pass), against the cells that the rules read and change, listed here from
their definitions (cans2d/bc/bdperx.f, bdsppx.f, bdsmnx.f, bdfrex.f, bdcnsx.f, bdfrdx.f):
in one pass each thread evaluates both faces' rules at its own cell, so no cell that a
rule changes may be read.  Every pair of rules, margins 1 to 4, from the smallest extent
a run takes to beyond where the two faces can meet.  CPU only."""
import ctypes as C
import itertools

import pytest

from utrip_gb300 import build, capi

KINDS = [capi.BD_NONE, capi.BD_PER, capi.BD_SPP, capi.BD_SPN, capi.BD_SMP, capi.BD_SMN,
         capi.BD_FRE, capi.BD_CNS, capi.BD_FRD]


@pytest.fixture(scope="module")
def probe():
    build.build()
    return C.CDLL(str(build.LIBDIR / build.PROBELIB))


def lower(kind, m, n):
    """{changed cell: cells its value is formed from}, 1-based, in front of any rule."""
    b = 1 + m
    src = {capi.BD_PER: lambda i: [n - m + 1 - i], capi.BD_SPP: lambda i: [b - 1 + i],
           capi.BD_SPN: lambda i: [b - 1 + i], capi.BD_SMP: lambda i: [b + i],
           capi.BD_SMN: lambda i: [b + i], capi.BD_FRE: lambda i: [b],
           capi.BD_CNS: lambda i: [], capi.BD_FRD: lambda i: [b, b + 1]}.get(kind)
    out = {} if src is None else {b - i: src(i) for i in range(1, m + 1)}
    if kind == capi.BD_SMN:
        out[b] = []
    return out


def independent(klo, khi, m, n):
    """Does no cell of a line that one pass reads change?"""
    lo = lower(klo, m, n)
    hi = {n + 1 - c: [n + 1 - s for s in srcs] for c, srcs in lower(khi, m, n).items()}
    reads = set()
    for c in set(lo) | set(hi):
        for s in hi.get(c, [c]):  # an upper rule's sources after the lower rule
            reads.update(lo[s] if s in lo else [s] if c in hi or s not in lo else [])
    return not reads & (set(lo) | set(hi))


@pytest.mark.parametrize("margin", [1, 2, 3, 4])
def test_one_pass_exactly_where_no_rule_reads_a_changed_cell(probe, margin):
    for n in range(2 * margin + 3, 3 * margin + 5):
        wide = 3 * margin + 20
        for lo, hi in itertools.product(KINDS, KINDS):
            want = independent(lo, hi, margin, n)
            for axis in (0, 1):
                kind = [capi.BD_NONE] * 4
                kind[2 * axis:2 * axis + 2] = [lo, hi]
                shape = (n, wide) if axis == 0 else (wide, n)
                got = probe.cans_probe_bc_one_pass(margin, *shape, (C.c_int * 4)(*kind))
                assert bool(got) == want, (margin, n, axis, lo, hi)
            if n >= 3 * margin + 2:
                assert want == ((lo, hi) != (capi.BD_PER, capi.BD_SMN))
