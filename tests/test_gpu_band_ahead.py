"""The one-column form of the band filter's coefficient kernel, which reads the
next 32 rows while it sums these, and the line between it and the two-column
form: grids of few columns with few modes take it (one to three modes a CTA),
with many modes or one mode on a narrow grid they do not.  Two steps of each
against the oracle, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx", [(160, 128), (544, 65), (160, 64), (192, 40)])
@pytest.mark.parametrize("band", [(5, 5), (2, 3), (2, 14), (3, 26), (2, 72)])
def test_bands_vs_oracle(cuda, orc, nz, nx, band):
    from kh_simulations_b200 import _lib
    from kh_simulations_b200._lib import Grid
    from kh_simulations_b200.config import derive, loads, step_params
    from kh_simulations_b200.run import KHRun

    cfg = loads(BASE + f"nz_override = {nz}\nnx_override = {nx}\nkz_bands = {band[0]}-{band[1]}\n", "bands")
    d = derive(cfg)
    run = KHRun(cfg)
    run.init()
    run.add_noise(1e-3, seed=8)
    s0 = run.state_numpy().copy()
    run.step(2)
    s = run.state_numpy()
    run.close()
    c, sn = np.empty((band[1] + 1, nz), np.float32), np.empty((band[1] + 1, nz), np.float32)
    _lib.check(_lib.load().ymkh_twiddles(nz, 0, band[1], c.ctypes.data_as(C.c_void_p), sn.ctypes.data_as(C.c_void_p)), "tw")
    want = orc.step(Grid(nx, nz, d.dx, d.dz), step_params(cfg, d), s0.copy(), 2, twiddles=(c, sn))
    assert np.array_equal(s.view(np.uint64), want.view(np.uint64))
