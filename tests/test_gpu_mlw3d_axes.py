"""One fast-policy 3-D step (plain, gravity, resistive) against the oracle on
stretched axes, whose corner weights need FP64 (equally spaced ones take integer
sums), with one stretched axis of the three, and on states with cells whose integer
sums are left to FP64; at extents around the tiles and z chunks.

Bound: as for equally spaced axes, an updated cell sums some 40 terms of a few
roundings each and the pressure is a difference of energies up to about 10 times
larger: 1e-13 of the largest value of each variable; cells the step keeps are equal."""
import numpy as np
import pytest

from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (18, 10, 5), (19, 11, 6), (5, 27, 68)]


@pytest.fixture(scope="module")
def oracle_lib():
    import oracle
    return oracle


def check(oracle_lib, s, shape, tiny=()):
    ref = setups.copy_state(s)
    dt, _ = oracle_lib.cfl_3d(s, ref, 0.4)
    oracle_lib.step_3d(s, ref, dt)
    got = setups.copy_state(s)
    drivers._step(s, got, dt)
    keep = np.ones(shape, dtype=bool)
    keep[(slice(1, -1),) * 3] = False
    for name, a, r, old in zip(s["names"], got, ref, s["state"]):
        floor = 1e-2 if name in tiny else 0.0
        assert np.max(np.abs(a - r)) <= 1e-13 * max(np.max(np.abs(r)), floor), name
        assert np.array_equal(a[keep], old[keep]), name


@pytest.mark.parametrize("axes", ["x", "y", "z", "xyz"])
@pytest.mark.parametrize("kind", ["plain", "gravity", "resistive"])
@pytest.mark.parametrize("shape", SHAPES)
def test_stretched_axes(oracle_lib, kind, axes, shape):
    s = setups.random_state_3d(*shape, seed=sum(shape))
    if kind == "gravity":
        s = setups.random_gravity(s, 3)
    if kind == "resistive":
        s = setups.random_resistivity(s, 4)
    s = dict(s)
    for a, n in zip("xyz", shape):  # spacings growing by 3 % a cell
        if a in axes:
            x = np.cumsum(0.01 * 1.03 ** np.arange(n))
            s["d" + a], _, s["d" + a + "m"] = setups.grdrdy(x)
    check(oracle_lib, s, shape)


@pytest.mark.parametrize("kind", ["plain", "gravity"])
@pytest.mark.parametrize("value", [1e-300, 5e-324, 1e-310, 0.0])
def test_components_out_of_the_integer_sums_range(oracle_lib, value, kind):
    """by and bz so small that they or their products leave the exponents of the
    integer sums, in half of the box: those corners and cells are summed in FP64."""
    shape = (19, 11, 9)
    s = setups.random_state_3d(*shape, seed=8)
    if kind == "gravity":
        s = setups.random_gravity(s, 3)
    for name in ("by", "bz"):
        s["state"][s["names"].index(name)][:10] = value
    check(oracle_lib, s, shape, tiny=("by", "bz"))
