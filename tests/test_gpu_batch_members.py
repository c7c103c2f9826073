"""What happens to a batch when its members are used between its steps: a
member given a new state, stepped alone, or given new parameters carries on
from there, bit for bit as a run alone."""
import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

# column stages as one kernel (64 rows), as separate ones (40 rows), none
TEXTS = ["nz_override = 64\nnx_override = 96\nhyp_diff = 5e-5\nkz_suppress_hi = 9\n",
         "nz_override = 40\nnx_override = 64\nhyp_diff = 5e-5\n",
         "nz_override = 32\nnx_override = 130\n"]


def _run(text):
    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    r = KHRun(loads(BASE + text))
    r.init()
    return r


def _state(text, steps, start=None):
    """State after `steps` steps alone from `start` (or the initial state)."""
    r = _run(text)
    if start is not None:
        r.set_state(start)
    r.step(steps)
    out = r.state_numpy()
    r.close()
    return out


def _batch(runs):
    from kh_simulations_b200.batch import KHBatch

    b = KHBatch()
    for r in runs:
        b.add(r)
    return b


@pytest.mark.parametrize("first", [3, 4])  # odd: the members are in their second buffers
@pytest.mark.parametrize("graphs", [False, True])
def test_member_state_set_between_batch_steps(cuda, first, graphs):
    import torch

    st = torch.cuda.Stream() if graphs else None
    runs = [_run(t) for t in TEXTS]
    b = _batch(runs)
    b.step(first, st)
    torch.cuda.synchronize()
    new = [_state(t, 7) for t in TEXTS]
    for i in (0, 1):
        runs[i].set_state(new[i])
    torch.cuda.synchronize()
    b.step(6, st)
    torch.cuda.synchronize()
    for i, (t, r) in enumerate(zip(TEXTS, runs)):
        want = _state(t, 6, new[i]) if i < 2 else _state(t, first + 6)
        assert np.array_equal(r.state_numpy(), want), t
    b.close()
    for r in runs:
        r.close()


@pytest.mark.parametrize("first", [2, 3])
def test_members_stepped_alone_between_batch_steps(cuda, first):
    import torch

    runs = [_run(t) for t in TEXTS]
    b = _batch(runs)
    b.step(first)
    runs[0].step(1)
    runs[1].step(3)
    b.step(5)
    runs[0].init()
    b.step(2)
    torch.cuda.synchronize()
    for t, r, n in zip(TEXTS, runs, (2, first + 10, first + 7)):
        assert np.array_equal(r.state_numpy(), _state(t, n)), t
    b.close()
    for r in runs:
        r.close()
