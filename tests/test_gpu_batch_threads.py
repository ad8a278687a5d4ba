"""Batches of several host threads, each with its own stream, share the kernels' per-device
launch data: started at the same time they end as one after the other, to the bit, on
every device there is."""
import threading

import numpy as np
import pytest

from utrip_gb300 import capi, setups

pytestmark = pytest.mark.gpu


def advance(k, exact, out, device=0):
    import torch
    torch.cuda.set_device(device)
    cases = [setups.random_state(40 + 3 * k, 36 + q, seed=k + q, solver="mlw_m3")
             for q in range(3)]
    b = capi.Batch(cases, exact=exact)
    for g, s in enumerate(cases):
        b.push(g, s["state"])
    b.start(nstop=20, safety=0.3, dtmin=1e-10)
    b.advance(20)
    out[k] = [b.pull(g) for g in range(3)]
    b.close()


@pytest.mark.parametrize("exact", [False, True])
def test_threads(gpu, exact):
    together, alone = {}, {}
    threads = [threading.Thread(target=advance, args=(k, exact, together)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    import torch
    for device in range(torch.cuda.device_count()):
        for k in range(4):
            advance(k, exact, alone, device)
            for a, b in zip(together[k], alone[k]):
                assert all(np.array_equal(x, y) for x, y in zip(a, b))
    torch.cuda.set_device(0)
