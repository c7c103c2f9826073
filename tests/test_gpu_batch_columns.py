"""Which members of a batch share the one column kernel: kernels launched a step
on both sides of each line of the rule, and every member bit for bit as alone
either way."""
import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

KZ0 = "suppress_kz0 = 1\n"


def _bands(modes):
    return f"kz_suppress_hi = {modes + 1}\n"  # modes 2 .. modes + 1


# four members; launches a step besides the FCT and Maxwell: 1 shared, or 4 x the member's own
CASES = [
    (256, 64, _bands(24), 1),
    (256, 64, _bands(25), 8),
    (160, 40, _bands(30), 8),
    (128, 64, _bands(40), 1),
    (64, 64, KZ0, 1),
    (128, 64, KZ0, 4),
    (128, 64, KZ0 + "hyp_diff = 5e-5\n", 1),
    (256, 64, KZ0 + _bands(40), 1),
    (512, 64, KZ0 + _bands(40), 12),
    (512, 64, KZ0 + _bands(14), 1),
    (512, 64, "hyp_diff = 5e-5\n", 4),
]


@pytest.mark.parametrize("nz,nx,text,launches", CASES)
def test_shared_column_kernel(cuda, nz, nx, text, launches):
    import torch

    from kh_simulations_b200 import _lib
    from kh_simulations_b200.batch import KHBatch
    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    runs = [KHRun(loads(BASE + f"nz_override = {nz}\nnx_override = {nx}\n" + text)) for _ in range(5)]
    for r in runs:
        r.init()
    alone = runs.pop()
    b = KHBatch(graph_steps=0)
    for r in runs:
        b.add(r)
    b.step(2)
    n0 = _lib.launch_count()
    b.step(1)
    assert _lib.launch_count() - n0 == 2 + launches
    torch.cuda.synchronize()
    alone.step(3)
    for r in runs:
        assert np.array_equal(r.state_numpy(), alone.state_numpy())
    b.close()
    for r in runs + [alone]:
        r.close()
