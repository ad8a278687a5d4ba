"""One step of the fast-policy Riemann solvers against the oracle on rough states
that reach every branch of their fluxes: supersonic faces of both signs, faces
between and outside the Alfven waves on both sides, a vanishing normal field
(bx = 0), a vanishing transverse field, equal states on both sides.

Bound: the flux is some 200 operations whose worst denominators (the star
states', the wave systems' determinants) are above 1e-3 of their terms on these
states, so a few hundred roundings times 1e3 in the few worst cells: 1e-10 of
each variable's largest value."""
import numpy as np
import pytest

from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle_lib():
    import oracle
    return oracle


def rough(solver, shape, seed, kind):
    s = setups.random_state_3d(*shape, seed=seed, solver=solver)
    rng = np.random.default_rng(seed)
    b = setups.SQ4PI * setups.B_UNIT[solver]
    speed = 4.0 if kind == "supersonic" else 0.7
    f = {"ro": rng.uniform(0.3, 2.0, shape), "pr": rng.uniform(0.2, 1.5, shape)}
    for k in ("vx", "vy", "vz"):
        f[k] = speed * rng.uniform(-1.0, 1.0, shape)
    for k in ("bx", "by", "bz"):
        f[k] = b * rng.uniform(-1.0, 1.0, shape)
    if kind == "no_normal":
        f["bx"][...] = 0.0
    if kind == "no_field":
        f["bx"][...] = f["by"][...] = f["bz"][...] = 0.0
    if kind == "blocks":  # equal neighbours, jumps between them
        for k in f:
            f[k] = np.repeat(f[k][::4], 4, axis=0)[: shape[0]]
    s["state"] = [np.asfortranarray(f[k]) for k in s["names"]]
    return s


CASES = [("hlld_3d", k) for k in ("subsonic", "supersonic", "no_normal", "no_field", "blocks")] + \
    [("roe_m_3d", k) for k in ("subsonic", "supersonic", "blocks")]


@pytest.mark.parametrize("solver,kind", CASES)
@pytest.mark.parametrize("shape", [(14, 11, 10), (33, 8, 9)])
def test_one_step_against_oracle(oracle_lib, solver, kind, shape):
    s = rough(solver, shape, sum(shape), kind)
    ref = setups.copy_state(s)
    dt, _ = oracle_lib.cfl_3d(s, ref, 0.1)
    oracle_lib.step_3d(s, ref, dt)
    got = setups.copy_state(s)
    drivers._step(s, got, dt)
    for name, a, r in zip(s["names"], got, ref):
        assert np.isfinite(r).all(), name
        assert np.max(np.abs(a - r)) <= 1e-10 * max(np.max(np.abs(r)), 1e-3), (name, kind)
