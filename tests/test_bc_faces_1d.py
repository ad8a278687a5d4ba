"""Where the two faces' rules of a 1-D line meet (cans::bc_faces_meet, against the cells
that the rules read and change; CPU), and the loop on a cluster of blocks there: periodic
faces against zeroed ones, mirrored ones that reach the other face, and periodic faces
with the chkdav floor, bit for bit the oracle's loop (exact policy), alone and in a
group."""
import ctypes as C
import itertools

import numpy as np
import pytest

from utrip_gb300 import build, capi, drivers, setups

NONE, PER, SPP, SPN, SMP, SMN, FRE, CNS, FRD = (
    capi.BD_NONE, capi.BD_PER, capi.BD_SPP, capi.BD_SPN, capi.BD_SMP, capi.BD_SMN, capi.BD_FRE,
    capi.BD_CNS, capi.BD_FRD)


def cells(kind, m, n):
    """Read and changed cells (1-based) of a rule on the lower face."""
    b = 1 + m
    i = range(1, m + 1)
    reads = {PER: {n - m + 1 - k for k in i}, SPP: {b - 1 + k for k in i},
             SPN: {b - 1 + k for k in i}, SMP: {b + k for k in i}, SMN: {b + k for k in i},
             FRE: {b}, FRD: {b, b + 1}}.get(kind, set())
    changes = set() if kind == NONE else {b - k for k in i} | ({b} if kind == SMN else set())
    return reads, changes


@pytest.mark.parametrize("margin", [1, 2, 3, 4])
def test_faces_meet_where_one_reads_what_the_other_changes(margin):
    build.build()
    probe = C.CDLL(str(build.LIBDIR / build.PROBELIB))
    kinds = [NONE, PER, SPP, SPN, SMP, SMN, FRE, CNS, FRD]
    for n in range(2 * margin + 2, 3 * margin + 6):
        for lo, hi in itertools.product(kinds, kinds):
            rl, cl = cells(lo, margin, n)
            rh, ch = ({n + 1 - c for c in s} for s in cells(hi, margin, n))
            want = bool(rl & ch) or bool(rh & cl)
            assert bool(probe.cans_probe_bc_faces_meet(margin, n, lo, hi)) == want, (n, lo, hi)


def make(ix, margin, pairs, seed):
    s = setups.random_state_1d(ix, seed=seed)
    s["margin"] = margin
    s["safety"] = 0.1
    s["bc"] = [(v, f, pairs[v][f], 0.5) for f in (0, 1) for v in range(5)]
    return s


MEET = [(PER, PER), (PER, PER), (PER, SMN), (SMN, PER), (PER, SMN)]
FLIPPED = [(SPP, SPP), (SPP, SPP), (SMN, PER), (SMP, SMN), (SMN, SMN)]
PERIODIC = [(PER, PER)] * 5
# 10 and 12 cells: two blocks whose mirrored faces reach each other's cells at margin 3
SIZES = [(70, 1), (71, 2), (130, 3), (10, 3), (12, 3), (1026, 1)]


def against_oracle(oracle_lib, cases, nstep, events):
    runs = []
    for s in cases:
        run = drivers.make_run(s, exact=True)
        run.push(s["state"])
        run.start(tend=1e30, nstop=nstep, safety=s["safety"], dtmin=s["dtmin"])
        runs.append(run)
    if len(runs) > 1:
        capi.Run.advance_group(runs, nstep)
    else:
        runs[0].advance(nstep)
    for s, run in zip(cases, runs):
        ref = setups.copy_state(s)
        if events:
            t_ref, n_floor = 0.0, 0
            for _ in range(nstep):
                one = {k: v for k, v in s.items() if k != "floor"}
                t_ref, _, merr, _ = oracle_lib.run_1d(one, ref, 1, t0=t_ref)
                assert merr == 0
                n_floor += oracle_lib.chkdav_state(s, ref)
            assert n_floor > 0 or len(ref[0]) < 70  # the smallest may hold none
        else:
            t_ref, _, merr, _ = oracle_lib.run_1d(s, ref, nstep)
            assert merr == 0
        assert all(np.isfinite(a).all() for a in ref)
        st = run.query()
        got = run.pull()
        run.close()
        assert (st.t, st.ns, st.merr) == (t_ref, nstep, 0)
        for name, a, b in zip(s["names"], got, ref):
            assert np.array_equal(a, b), name
        if events:
            assert st.n_floor == n_floor


@pytest.mark.gpu
@pytest.mark.parametrize("group", [1, 3])
@pytest.mark.parametrize("pairs", [MEET, FLIPPED], ids=["meet", "flipped"])
@pytest.mark.parametrize("ix,margin", SIZES)
def test_rules_that_meet(oracle_lib, gpu, ix, margin, pairs, group):
    against_oracle(oracle_lib, [make(ix, margin, pairs, k) for k in range(group)], 6, False)


@pytest.mark.gpu
@pytest.mark.parametrize("group", [1, 3])
@pytest.mark.parametrize("pairs", [PERIODIC, MEET], ids=["periodic", "meet"])
@pytest.mark.parametrize("ix,margin", SIZES)
def test_periodic_faces_with_the_floor(oracle_lib, gpu, ix, margin, pairs, group):
    cases = [make(ix, margin, pairs, k) for k in range(group)]
    for s in cases:
        s["floor"] = 0.65  # pressures start at 0.6: cells at both faces are floored
    against_oracle(oracle_lib, cases, 6, True)
