"""One 3-D step of the double-float policy against the oracle on equally spaced axes
(corner weights as float corrections) and on stretched ones (weights in
double-float), on both tiles, at extents around the tiles and z chunks.

Bound: an updated cell sums some 40 terms of a few roundings of 2^-46 each, and the
pressure is a difference of energies up to about 10 times larger: 40 x 4 x 10 x
2^-46 = 2.3e-11 of the largest value of each variable; cells the step keeps are equal."""
import numpy as np
import pytest

from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 4), (18, 10, 5), (19, 11, 6), (18, 18, 7), (19, 19, 5), (5, 27, 68)]


@pytest.mark.parametrize("axes", ["", "x", "y", "z", "xyz"])
@pytest.mark.parametrize("tile", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_one_step_against_oracle(oracle_lib, gpu, shape, tile, axes):
    s = dict(setups.random_state_3d(*shape, seed=sum(shape)))
    for a, n in zip("xyz", shape):  # spacings growing by 3 % a cell
        if a in axes:
            x = np.cumsum(0.01 * 1.03 ** np.arange(n))
            s["d" + a], _, s["d" + a + "m"] = setups.grdrdy(x)
    ref = setups.copy_state(s)
    dt, _ = oracle_lib.cfl_3d(s, ref, 0.4)
    oracle_lib.step_3d(s, ref, dt)
    run = drivers.make_run(s, tile=tile, df64=True)
    run.push(s["state"])
    run.step(dt, apply_bc=False)
    got = run.pull()
    run.close()
    keep = np.ones(shape, dtype=bool)
    keep[(slice(1, -1),) * 3] = False
    for name, a, r, old in zip(s["names"], got, ref, s["state"]):
        assert np.max(np.abs(a - r)) <= 2.3e-11 * np.max(np.abs(r)), name
        assert np.array_equal(a[keep], old[keep]), name
