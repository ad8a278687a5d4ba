"""One fast-policy 3-D step (plain, with gravity, resistive) on every tile against
the oracle, at extents around the tiles' edges: the smallest array, whole tiles,
one cell more and one less, and z chunks that do not divide.

Bound: an updated cell sums some 40 terms of a few roundings each, and the
pressure is a difference of energies up to about 10 times larger, so 1e-13 of
the largest value of each variable; cells the step keeps are equal."""
import numpy as np
import pytest

from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (4, 4, 4), (18, 10, 5), (17, 9, 4), (19, 11, 6), (34, 14, 7), (21, 27, 68), (5, 40, 35)]


@pytest.fixture(scope="module")
def oracle_lib():
    import oracle
    return oracle


def make(kind, shape, seed):
    s = setups.random_state_3d(*shape, seed=seed)
    if kind == "gravity":
        return setups.random_gravity(s, seed + 1)
    if kind == "resistive":
        return setups.random_resistivity(s, seed + 1)
    return s


@pytest.mark.parametrize("kind", ["plain", "gravity", "resistive"])
@pytest.mark.parametrize("tile", [0, 1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_one_step_against_oracle(oracle_lib, kind, tile, shape):
    s = make(kind, shape, 11)
    ref = setups.copy_state(s)
    dt, _ = oracle_lib.cfl_3d(s, ref, 0.4)
    oracle_lib.step_3d(s, ref, dt)
    if min(shape) < 4:  # below a run handle's two frames: the drop-in call
        got = setups.copy_state(s)
        drivers._step(s, got, dt)
    else:
        run = drivers.make_run(s, tile=tile)
        run.push(s["state"])
        run.step(dt, apply_bc=False)
        got = run.pull()
        run.close()
    inner = (slice(1, -1),) * 3
    for name, a, r, old in zip(s["names"], got, ref, s["state"]):
        assert np.max(np.abs(a - r)) <= 1e-13 * np.max(np.abs(r)), (name, shape, tile)
        keep = np.ones(shape, dtype=bool)
        keep[inner] = False
        assert np.array_equal(a[keep], old[keep]), name


@pytest.mark.parametrize("tile", [0, 1, 2])
def test_loop_time_steps_against_oracle(oracle_lib, tile):
    """The CFL of the loop (reduced as a key in the step's epilogue): five
    iterations reach the oracle's time."""
    s = setups.random_state_3d(23, 21, 19, seed=5)
    ref = setups.copy_state(s)
    t_ref, ns, _, _ = oracle_lib.run_3d(s, ref, 5)
    run = drivers.make_run(s, tile=tile)
    st = setups.copy_state(s)
    t, n, merr, nexec = drivers.run_resident(s, st, 5, run=run)
    run.close()
    assert (n, merr, nexec) == (ns, 0, 5) and abs(t - t_ref) <= 1e-13 * t_ref
    for a, r in zip(st, ref):
        assert np.max(np.abs(a - r)) <= 1e-12 * np.max(np.abs(r))
