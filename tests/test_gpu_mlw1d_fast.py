"""The fast-policy 1-D step (mlw_m) against the oracle: one step at extents around
the cluster's blocks (one block, unequal shares, the block of whole warps, several
passes of a block) on equal and stretched spacings, and the loop's CFL minimum,
which the blocks exchange as keys.

Bound: an updated cell sums some 20 terms of a few roundings each and the
pressure is a difference of energies up to about 10 times larger: 1e-13 of the
largest value of each variable; the loop's time is a sum of minima that agree to a
few roundings each: 1e-13 a step."""
import numpy as np
import pytest

import oracle
from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu


def make(ix, axes):
    s = setups.random_state_1d(ix, seed=ix)
    if axes == "stretched":
        s["dx"], _, s["dxm"] = setups.grdrdy(np.cumsum(0.01 * 1.03 ** (np.arange(ix) % 100)))
    return s


@pytest.mark.parametrize("axes", ["equal", "stretched"])
@pytest.mark.parametrize("ix", [6, 7, 9, 35, 66, 67, 130, 515, 1026, 4099])
def test_one_step_against_oracle(oracle_lib, gpu, ix, axes):
    s = make(ix, axes)
    ref = setups.copy_state(s)
    dt, _ = oracle.cfl_m_1d(0.4, 1e-10, s["gm"], s["bx"], *ref, s["dx"])
    oracle.mlw_m_1d(*ref, s["bx"], s["bxm"], dt, s["qav"], s["gm"], s["dx"], s["dxm"])
    got = setups.copy_state(s)
    gpu.set_exact(False)
    drivers._step(s, got, dt)
    for name, a, r, old in zip(s["names"], got, ref, s["state"]):
        assert np.max(np.abs(a - r)) <= 1e-13 * np.max(np.abs(r)), name
        assert a[0] == old[0] and a[-1] == old[-1], name


@pytest.mark.parametrize("ix", [6, 35, 67, 130, 1026, 4099])
def test_loop_time_against_oracle(oracle_lib, gpu, ix):
    s = make(ix, "equal")
    s["safety"] = 0.2
    ref = setups.copy_state(s)
    t_ref, ns, _, _ = oracle.run_1d(s, ref, 5)
    gpu.set_exact(False)
    st = setups.copy_state(s)
    t, n, merr, nexec = drivers.run_resident(s, st, 5)
    assert (n, merr, nexec) == (ns, 0, 5) and abs(t - t_ref) <= 5e-13 * t_ref
