"""Batches of narrow grids take narrower strips than those of wide ones; every
member ends as it does alone, bit for bit, whatever width the batch takes:
sets of members around the rule's edges (26 and 58 columns, where a strip is
full), copied by TMA and by element, narrow and wide together."""
import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

WALLS = "run_mode = 0\n"
SETS = {
    "one 32-wide strip": [(96, 26, ""), (33, 25, WALLS), (40, 4, "")],
    "one 64-wide strip": [(96, 58, ""), (64, 27, WALLS), (50, 48, "warm_T = 0.01\n")],
    "128-wide": [(96, 60, ""), (96, 120, WALLS), (64, 130, "")],
    "narrow and wide": [(96, 8, ""), (96, 34, WALLS), (64, 68, ""), (64, 69, WALLS)],
    "narrow, one wide": [(300, 16, "")] * 3 + [(32, 128, "")],
}


def _run(nz, nx, text):
    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    r = KHRun(loads(BASE + f"nz_override = {nz}\nnx_override = {nx}\n" + text))
    r.init()
    return r


@pytest.mark.parametrize("name", SETS)
def test_batch_of_narrow_grids_equals_alone(cuda, name):
    import torch

    from kh_simulations_b200.batch import KHBatch

    runs = [_run(*m) for m in SETS[name]]
    b = KHBatch()
    for r in runs:
        b.add(r)
    b.step(5)
    torch.cuda.synchronize()
    b.check()
    for m, r in zip(SETS[name], runs):
        alone = _run(*m)
        alone.step(5)
        assert np.array_equal(r.state_numpy(), alone.state_numpy()), m
        alone.close()
    b.close()
    for r in runs:
        r.close()
