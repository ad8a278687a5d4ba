"""The 2-D boundary program at the extents where the faces' rules meet (2 margin + 2 ..
3 margin + 2 cells, the smallest a run takes) against the oracle's, axis by axis and rule
by rule: the same bits, for every pair of rules that reads what the other face changes, in
a run's step, its loops (with and without chkdav) and a batch (exact policy)."""
import numpy as np
import pytest

from utrip_gb300 import capi, drivers, setups

pytestmark = pytest.mark.gpu

PER, SPP, SPN, SMP, SMN, FRE, CNS, FRD = (capi.BD_PER, capi.BD_SPP, capi.BD_SPN, capi.BD_SMP,
                                          capi.BD_SMN, capi.BD_FRE, capi.BD_CNS, capi.BD_FRD)
PAIRS = [(SMP, SMN), (SMN, SMN), (SMP, SPP), (SMN, FRD), (SPP, SMN), (SPN, SMN), (PER, SMN),
         (SMN, PER), (PER, PER), (SMP, FRE), (SMN, CNS), (FRD, SMP)]


def make(margin, shape, first, pairs=PAIRS, keep=()):
    """A state whose variables take `pairs` in turn on both axes, from `first` on; those
    of `keep` (the density and pressure of a loop) are mirrored."""
    s = setups.random_state(*shape, seed=first, solver="mlw_m3", margin=margin)
    s["bc"] = []
    for v in range(len(s["state"])):
        for axis in (0, 1):
            lo, hi = (SPP, SPP) if v in keep else pairs[(first + v + 5 * axis) % len(pairs)]
            s["bc"] += [(v, 2 * axis, lo, 0.7), (v, 2 * axis + 1, hi, 0.9)]
    return s


def shapes(margin):
    return [(margin, shape) for n in range(2 * margin + 2, 3 * margin + 3)
            for shape in ((n, n), (n, 40), (70, n))]


@pytest.mark.parametrize("first", range(0, len(PAIRS), 3))
@pytest.mark.parametrize("margin,shape", [c for m in (1, 2, 3, 4) for c in shapes(m)])
def test_fill(oracle_lib, gpu, margin, shape, first):
    s = make(margin, shape, first)
    run = drivers.make_run(s, exact=True)
    got = []
    for fill in (False, True):
        run.push(s["state"])
        run.step(1e-5, apply_bc=fill)
        got.append(run.pull())
    run.close()
    want = [a.copy(order="F") for a in got[0]]
    oracle_lib.apply_bc_program(want, s["bc"], margin, s)
    for name, a, b in zip(s["names"], got[1], want):
        assert np.array_equal(a, b, equal_nan=True), name


@pytest.mark.parametrize("floor", [None, 1e-3])
@pytest.mark.parametrize("margin,shape", [c for m in (1, 2, 3) for c in shapes(m)])
def test_loops_and_batch(oracle_lib, gpu, margin, shape, floor):
    s = make(margin, shape, 1, keep=(0, 1))
    s["safety"], s["floor"] = 0.1, floor
    ref = setups.copy_state(s)
    t_ref, ns, merr_ref, _ = oracle_lib.run_2d(s, ref, 4)
    assert merr_ref == 0 and all(np.isfinite(a).all() for a in ref)
    st = setups.copy_state(s)
    t, n, merr, _ = drivers.run_resident(s, st, 4, exact=True)
    assert (t, n, merr) == (t_ref, ns, 0)
    for name, a, b in zip(s["names"], st, ref):
        assert np.array_equal(a, b), name
    if floor is not None or min(shape) < 2 * margin + 3:
        return
    batch = capi.Batch([s, make(margin, (40, 50), 2, keep=(0, 1))], exact=True)
    batch.push(0, s["state"])
    batch.push(1, make(margin, (40, 50), 2, keep=(0, 1))["state"])
    batch.start(nstop=4, safety=s["safety"], dtmin=s["dtmin"])
    batch.advance(4)
    got = batch.pull(0)
    batch.close()
    for name, a, b in zip(s["names"], got, ref):
        assert np.array_equal(a, b), name
