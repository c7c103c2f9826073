"""The strip width that a run takes by itself, at the edges of the rule: narrow
grids stay with 32-wide strips however tall they are (the 128-wide form took up
to three times as long there)."""
import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu


def _run(nz, nx, text=""):
    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    r = KHRun(loads(BASE + f"nz_override = {nz}\nnx_override = {nx}\n" + text))
    r.init()
    return r


@pytest.mark.parametrize("nz,nx,width", [(128, 4, 32), (512, 16, 32), (2048, 48, 32), (128, 63, 32), (128, 64, 128),
                                         (127, 64, 32), (127, 127, 32), (32, 128, 128)])
@pytest.mark.parametrize("walls", ["", "run_mode = 0\n"])
def test_default_strip_width(cuda, nz, nx, width, walls):
    from kh_simulations_b200 import _lib

    r, split = _run(nz, nx, walls), _run(nz, nx, walls)
    assert r.fct_shape()[0] == width
    _lib.check(split.lib.ymkh_set_fct_mode(split.ctx, _lib.FCT_SPLIT), "ymkh_set_fct_mode")
    r.step(3)
    split.step(3)
    assert np.array_equal(r.state_numpy(), split.state_numpy())
    r.close()
    split.close()
