"""push and pull of a run: states in page-locked arrays (one launch below 1 MB, copies
beyond), in pageable ones and in a mixture of both give the same bits, at sizes
around the launch's blocks and its limit; and a 1-D run started again without a
wait steps as a fresh one."""
import numpy as np
import pytest
import torch

from utrip_gb300 import drivers, setups

pytestmark = pytest.mark.gpu


def pinned(a):
    p = torch.empty(tuple(reversed(a.shape)), dtype=torch.float64, pin_memory=True).numpy().T
    p[...] = a
    return p


def keep(a, k, which):
    return pinned(a) if which == "pinned" or (which == "mixed" and k % 2) else a.copy(order="F")


SETUPS = {f"1d_{n}": (lambda n=n: setups.random_state_1d(n, seed=n)) for n in (6, 256, 257, 1026, 15000)}
SETUPS.update({f"2d_{a}x{b}": (lambda a=a, b=b: setups.random_state(a, b, seed=a))
               for a, b in ((5, 7), (120, 121), (121, 121))})  # just below and above 1 MB
SETUPS["3d"] = lambda: setups.random_state_3d(25, 25, 26, seed=3)


@pytest.mark.parametrize("which", ["pageable", "pinned", "mixed"])
@pytest.mark.parametrize("name", list(SETUPS))
def test_push_pull(gpu, name, which):
    s = SETUPS[name]()
    run = drivers.make_run(s)
    src = [keep(a, k, which) for k, a in enumerate(s["state"])]
    out = [keep(np.full_like(a, np.nan), k, which) for k, a in enumerate(s["state"])]
    run.push(src)
    run.pull(out)
    run.close()
    for a, b in zip(out, s["state"]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("which", ["pageable", "pinned"])
def test_restarted_run_steps_as_a_fresh_one(gpu, which):
    s = setups.random_state_1d(1026, seed=9)
    src = [keep(a, k, which) for k, a in enumerate(s["state"])]
    got = []
    run = drivers.make_run(s)
    for iters in (7, 30, 30):  # the first leaves another state, time and dt behind
        run.push(src)
        run.start(nstop=10 ** 9, safety=s["safety"], dtmin=s["dtmin"])
        run.advance(iters)
        got.append((run.pull(), run.query().t))
    run.close()
    assert got[1][1] == got[2][1] and got[0][1] < got[1][1]
    for a, b in zip(got[1][0], got[2][0]):
        assert np.array_equal(a, b)


def test_a_started_run_has_taken_its_arrays(gpu):
    """The page-locked arrays may be filled again once start has returned, also with
    work of an earlier loop in front of the push."""
    s = setups.random_state_1d(1026, seed=9)
    src = [pinned(a) for a in s["state"]]
    run = drivers.make_run(s)
    for _ in range(3):
        for p, a in zip(src, s["state"]):
            p[...] = a
        run.push(src)
        run.start(nstop=10 ** 9, safety=s["safety"], dtmin=s["dtmin"])
        for p in src:
            p[...] = -1.0
        run.advance(2000)
    assert run.query().merr == 0 and np.all(run.pull()[0] > 0.0)
    run.push(src)
    for p, a in zip(src, s["state"]):
        p[...] = a
    run.push(src)
    out = run.pull()
    run.close()
    for a, b in zip(out, s["state"]):
        assert np.array_equal(a, b)
