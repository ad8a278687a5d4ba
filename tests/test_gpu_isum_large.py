"""The fast 2-D and 3-D steps on states whose energy fluxes lie at the upper end of the
integer sums' exponents (velocities and fields of 2^333 .. 2^338, pressures of their
square: fluxes of 2^999 .. 2^1014, which the corrector sums at up to 32 times their
value), below it, across it and beyond it, where the sums are FP64's: against the oracle,
to the bound of the ordinary states, 1e-13 of each variable's largest value.  A scale by
a power of two is exact, so the oracle's step is that of the unscaled state but for the
viscosity's threshold."""
import numpy as np
import pytest

from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu

POWER = {"pr": 2, "vx": 1, "vy": 1, "vz": 1, "bx": 1, "by": 1, "bz": 1, "az": 1}


@pytest.mark.parametrize("exponent", [333, 336, 337, 338])
@pytest.mark.parametrize("kind", ["mlw_m3", "mlw_m", "mlw_m_3d"])
def test_large_fluxes(oracle_lib, gpu, kind, exponent):
    if kind == "mlw_m_3d":
        s = setups.random_state_3d(19, 18, 9, seed=2)
        cfl, step = oracle_lib.cfl_3d, oracle_lib.step_3d
    else:
        s = setups.random_state(70, 40, seed=2, solver=kind)
        cfl, step = oracle_lib.cfl_2d, oracle_lib.step_2d
    s["state"] = [a * 2.0 ** (exponent * POWER.get(k, 0)) for k, a in zip(s["names"], s["state"])]
    s["dtmin"] = 0.0
    ref = setups.copy_state(s)
    dt, _ = cfl(s, ref, 0.4)
    assert 0.0 < dt < 1.0
    step(s, ref, dt)
    got = setups.copy_state(s)
    gpu.set_exact(False)
    drivers._step(s, got, dt)
    for name, a, r in zip(s["names"], got, ref):
        assert np.isfinite(r).all()
        assert np.max(np.abs(a - r)) <= 1e-13 * np.max(np.abs(r)), name
