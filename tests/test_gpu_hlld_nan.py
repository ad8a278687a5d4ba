"""A cell that is not a number makes its neighbours so: the HLLD flux of a face with such
a state on either side is not a number in any component while the flow is subsonic, and
with such a state on the right side also where the flow comes from the left at supersonic
speed (the reference's max(cfl, cfr) takes the right speed then).  The fast flux compares
integers, where a NaN has an order, so each of its comparisons is reached here: NaNs of
both signs in each variable, a negative density (whose fast speed is not a number), on
both sides of faces of every axis.  The exact policy shows the same."""
import numpy as np
import pytest

from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu

CELL = (6, 5, 6)
MINUS_NAN = np.array([0xFFF8000000000000], dtype=np.uint64).view(np.float64)[0]


def uniform(bad_var, bad, axis=0, speed=0.1):
    """A uniform box moving along `axis` with one bad cell."""
    s = setups.random_state_3d(13, 12, 14, seed=1, solver="hlld_3d")
    val = dict(ro=1.0, pr=0.6, vx=0.05, vy=0.04, vz=0.03, bx=0.3, by=0.2, bz=0.25)
    val["v" + "xyz"[axis]] = speed
    s["state"] = [np.full((13, 12, 14), val[k], order="F") for k in s["names"]]
    s["state"][s["names"].index(bad_var)][CELL] = bad
    return s


def step(gpu, s, exact):
    got = setups.copy_state(s)
    gpu.set_exact(exact)
    try:
        drivers._step(s, got, 1e-3)
    finally:
        gpu.set_exact(False)
    return dict(zip(s["names"], got))


def neighbour(axis, d):
    return tuple(c + (d if a == axis else 0) for a, c in enumerate(CELL))


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("bad", [np.nan, MINUS_NAN], ids=["nan", "minus_nan"])
@pytest.mark.parametrize("var", ["ro", "pr", "vx", "vy", "vz", "by", "bz"])
def test_subsonic(gpu, var, bad, exact):
    got = step(gpu, uniform(var, bad), exact)
    for axis in range(3):
        for d in (-1, 1):
            for k in ("ro", "pr", "vx", "vy", "vz"):
                assert np.isnan(got[k][neighbour(axis, d)]), (axis, d, k)


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("var,bad", [("pr", np.nan), ("pr", MINUS_NAN), ("ro", -1.0)],
                         ids=["nan", "minus_nan", "negative"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_supersonic_from_the_left(gpu, axis, var, bad, exact):
    """The upstream neighbour's face has the bad state on its right."""
    got = step(gpu, uniform(var, bad, axis, 9.0), exact)
    for k in ("ro", "pr", "vx", "vy", "vz"):
        assert np.isnan(got[k][neighbour(axis, -1)]), k
