"""A batch that holds equally spaced and stretched meshes: each run ends as in a batch
of its own, to the bit, in the fast policy too (its arithmetic is that of its own mesh),
and as the oracle's loop in the exact policy."""
import numpy as np
import pytest

from utrip_gb300 import capi, setups

pytestmark = pytest.mark.gpu


def run(shape, seed, solver, stretched):
    s = setups.random_state(*shape, seed=seed, solver=solver)
    if stretched:
        for a, n in zip("xy", shape):
            if a in stretched:
                x = np.cumsum(0.01 * 1.03 ** np.arange(n))
                s["d" + a], _, s["d" + a + "m"] = setups.grdrdy(x)
    return s


def advance(cases, exact, config):
    b = capi.Batch(cases, exact=exact)
    b.lib.cans_batch_set_config(b.h, config)
    for g, s in enumerate(cases):
        b.push(g, s["state"])
    b.start(nstop=12, safety=0.3, dtmin=1e-10)
    b.advance(15)
    out = [(b.query(g).t, b.query(g).ns, b.pull(g)) for g in range(len(cases))]
    b.close()
    return out


@pytest.mark.parametrize("config", [0, 1])
@pytest.mark.parametrize("solver", ["mlw_m3", "mlw_m"])
@pytest.mark.parametrize("exact", [False, True])
def test_runs_do_not_depend_on_their_company(oracle_lib, gpu, exact, solver, config):
    cases = [run((40, 36), 1, solver, ""), run((33, 70), 2, solver, "xy"),
             run((66, 48), 3, solver, ""), run((47, 29), 4, solver, "y"),
             run((100, 31), 5, solver, "")]
    together = advance(cases, exact, config)
    for s, (t, ns, state) in zip(cases, together):
        (t1, ns1, alone), = advance([s], exact, config)
        assert (t, ns) == (t1, ns1) == (t1, 12)
        for name, a, b in zip(s["names"], state, alone):
            assert np.array_equal(a, b), name
        if exact:
            s["safety"] = 0.3
            ref = setups.copy_state(s)
            assert oracle_lib.run_2d(s, ref, 12)[0] == t
            for name, a, b in zip(s["names"], state, ref):
                assert np.array_equal(a, b), name
