"""The 2-D boundary program of a run in one launch (x and y rules together) against
the oracle's, axis by axis and rule by rule: the same bits, for every kind of rule
drawn per variable and face, at margins 1 to 3 and extents from the smallest a run
takes.  The step in front of it is the exact policy's own.  In the loops and the batch
a program whose lower rule reads what the upper one zeroes gives the oracle's bits
too."""
import numpy as np
import pytest

from utrip_gb300 import capi, drivers, setups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("shape", [(12, 12), (13, 37), (70, 12), (131, 66)])
@pytest.mark.parametrize("solver,margin", [("mlw_m3", 1), ("mlw_m", 1), ("mlw_m3", 2), ("mlw_m3", 3),
                                           ("roe_m3", 3)])
def test_fill_is_the_oracles(oracle_lib, gpu, solver, margin, shape, seed):
    s = setups.random_state(*shape, seed=seed, solver=solver)
    rng = np.random.default_rng(seed * 10 + margin)
    s["margin"] = margin
    s["bc"] = [(v, f, int(rng.integers(0, 8)), float(rng.uniform(0.5, 1.0)))
               for v in range(len(s["state"])) for f in range(4)]
    run = drivers.make_run(s, exact=True)
    got = []
    for fill in (False, True):
        run.push(s["state"])
        run.step(1e-4, apply_bc=fill)
        got.append(run.pull())
    run.close()
    want = [a.copy(order="F") for a in got[0]]
    oracle_lib.apply_bc_program(want, s["bc"], margin, s)
    for name, a, b in zip(s["names"], got[1], want):
        assert np.array_equal(a, b, equal_nan=True), name


def mixed_setup(shape, axis):
    s = setups.random_state(*shape, seed=4, solver="mlw_m3")
    s["bc"] = [(v, f, k, q) for v, f, k, q in s["bc"] if (v, f // 2) != (2, axis)]
    s["bc"] += [(2, 2 * axis, capi.BD_PER, 0.0), (2, 2 * axis + 1, capi.BD_SMN, 0.0)]
    return s


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("shape", [(13, 37), (131, 66)])
def test_mixed_program_in_loops(oracle_lib, gpu, shape, axis):
    s = mixed_setup(shape, axis)
    ref = setups.copy_state(s)
    t_ref, ns, _, _ = oracle_lib.run_2d(s, ref, 12)
    st = setups.copy_state(s)
    t, n, merr, _ = drivers.run_resident(s, st, 12, exact=True)
    assert (t, n, merr) == (t_ref, ns, 0)
    batch = capi.Batch([s, mixed_setup((40, 50), 1 - axis)], exact=True)
    for g, q in enumerate((s, mixed_setup((40, 50), 1 - axis))):
        batch.push(g, q["state"])
    batch.start(nstop=12, safety=s["safety"], dtmin=s["dtmin"])
    batch.advance(12)
    got = batch.pull(0)
    batch.close()
    for name, a, b, c in zip(s["names"], st, ref, got):
        assert np.array_equal(a, b) and np.array_equal(c, b), name
