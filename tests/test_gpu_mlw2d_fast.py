"""One fast-policy 2-D step (both solvers; plain, gravity, resistive) against the
oracle on equally spaced axes, whose corner differences are integer sums, and on
stretched ones, whose weights need FP64, at extents around the strips, chunks and
segments of the marching block; and on states with cells that integer sums
leave to FP64.

Bound: an updated cell sums some 20 terms of a few roundings each and the
pressure is a difference of energies up to about 10 times larger: 1e-13 of the
largest value of each variable; cells the step keeps are equal."""
import numpy as np
import pytest

from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3), (4, 9), (34, 9), (33, 10), (35, 16), (66, 17), (100, 31), (37, 140)]


@pytest.fixture(scope="module")
def oracle_lib():
    import oracle
    return oracle


def stretch(s):
    """The axes with spacings growing by 3 % a cell."""
    out = dict(s)
    for a, n in zip("xy", s["state"][0].shape):
        x = np.cumsum(0.01 * 1.03 ** np.arange(n))
        out["d" + a], _, out["d" + a + "m"] = setups.grdrdy(x)
    return out


def make(solver, kind, axes, shape):
    s = setups.random_state(*shape, seed=sum(shape), solver=solver)
    if kind in ("gravity", "both"):
        s = setups.random_gravity(s, 3)
    if kind in ("resistive", "both"):
        s = setups.random_resistivity(s, 4, scale=0.002)
    return stretch(s) if axes == "stretched" else s


def check(oracle_lib, s, shape):
    ref = setups.copy_state(s)
    dt, _ = oracle_lib.cfl_2d(s, ref, 0.4)
    oracle_lib.step_2d(s, ref, dt)
    got = setups.copy_state(s)
    drivers._step(s, got, dt)
    keep = np.ones(shape, dtype=bool)
    keep[1:-1, 1:-1] = False
    for name, a, r, old in zip(s["names"], got, ref, s["state"]):
        assert np.max(np.abs(a - r)) <= 1e-13 * max(np.max(np.abs(r)), 1e-2), name
        assert np.array_equal(a[keep], old[keep]), name


@pytest.mark.parametrize("axes", ["uniform", "stretched"])
@pytest.mark.parametrize("kind", ["plain", "gravity", "resistive", "both"])
@pytest.mark.parametrize("solver", ["mlw_m3", "mlw_m"])
@pytest.mark.parametrize("shape", SHAPES)
def test_one_step_against_oracle(oracle_lib, solver, kind, axes, shape):
    if min(shape) < 4 and solver == "mlw_m" and axes == "stretched":
        pytest.skip("the same cells as mlw_m3's")
    check(oracle_lib, make(solver, kind, axes, shape), shape)


@pytest.mark.parametrize("value", [1e-300, 5e-324, 1e-310, 0.0])
def test_components_out_of_the_integer_sums_range(oracle_lib, value):
    """vz and bz so small that their products leave the exponents of the integer
    sums, in half of the box: those corners and cells are summed in FP64."""
    shape = (70, 40)
    s = make("mlw_m3", "plain", "uniform", shape)
    st = dict(zip(s["names"], s["state"]))
    for k in ("vz", "bz"):
        st[k][:35] = value * np.sign(st[k][:35])
        if value == 0.0:
            st[k][...] = 0.0
    check(oracle_lib, s, shape)
