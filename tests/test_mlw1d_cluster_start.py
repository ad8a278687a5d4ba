"""The blocks of a 1-D run's cluster write into each other's shared memory (halos, the
minimum's slots).  A block may do so only once the others run, which a cluster barrier
guarantees: the loop kernel has one in front of the first such write.  The order is read
in the source (a violation need not show in a result); on the GPU more runs than the
device holds at once, advanced one step a launch, so that clusters start at all times,
end bit for bit as the oracle's (exact policy)."""
from pathlib import Path

import numpy as np
import pytest

from utrip_gb300 import build, capi, drivers, setups


def test_a_cluster_barrier_stands_before_the_first_remote_write():
    text = (Path(build.CSRC) / "mlw1d.cu").read_text()
    body = text[text.index("void mlw1d_body("):text.index("k_mlw1d_group(")]
    assert body.index("cluster.sync()") < body.index("map_shared_rank(")


@pytest.mark.gpu
@pytest.mark.parametrize("ix,nruns", [(300, 200), (600, 150), (1100, 90)])
def test_many_clusters_one_step_a_launch(oracle_lib, gpu, ix, nruns):
    cases = [setups.random_state_1d(ix + k % 3, seed=k) for k in range(nruns)]
    runs = []
    for s in cases:
        run = drivers.make_run(s, exact=True)
        run.push(s["state"])
        run.start(tend=1e30, nstop=5, safety=0.2, dtmin=s["dtmin"])
        runs.append(run)
    for _ in range(5):
        capi.Run.advance_group(runs, 1)
    for s, run in zip(cases, runs):
        s["safety"] = 0.2
        ref = setups.copy_state(s)
        t_ref, ns, _, _ = oracle_lib.run_1d(s, ref, 5)
        st = run.query()
        got = run.pull()
        run.close()
        assert (st.t, st.ns, st.merr) == (t_ref, ns, 0)
        for name, a, b in zip(s["names"], got, ref):
            assert np.array_equal(a, b), name
