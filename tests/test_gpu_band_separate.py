"""The separate FP64 band kernels (band_coef_kernel, band_apply_kernel) at the
edges of their blocks, bit for bit: columns just past a 128-column block and no
multiple of one, rows that are no multiple of 32, bands of one mode, of exactly
a 16-mode block and of one more, several bands in one run, and rows past the
one-kernel form's 512.  Against the oracle where NZ is a multiple of 32 (the
reference's kernels and the oracle leave out the rows past the last whole warp
otherwise), else against the same sums in numpy with the last warp filled up
with zeros."""
import ctypes as C

import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

CASES = [
    (160, 200, "kz_bands = 5-40\n"),
    (161, 129, "kz_keep_max = 53\n"),
    (100, 257, "kz_bands = 7-7\n"),
    (250, 130, "kz_bands = 3-18\n"),
    (31, 127, "kz_bands = 2-4\n"),
    (544, 150, "kz_bands = 3-19\nkz_suppress_max = 2\nkz_suppress_hi = 7\n"),
    (1024, 130, "kz_bands = 300-333, 9-9\nsuppress_kz0 = 1\n"),
]
# the filtered arrays: every field but Az1, and n, px, pz and Q2, Q3 of both beams
FILTERED = [a for a in range(24) if a not in (9, 15, 21)]


def _subtract_band(v, lo, hi, cos, sin):
    """v[z, x] without the modes lo..hi, summed as the kernels sum."""
    nz, nx = v.shape
    inv2 = float(np.float32(2.0) / np.float32(nz))
    rows = -(-nz // 32) * 32

    def coef(w):
        a = np.zeros((rows, nx))
        a[:nz] = v * w[:, None].astype(np.float64)
        a = a.reshape(rows // 32, 32, nx)
        for h in (16, 8, 4, 2, 1):  # the warps' shuffle trees
            a = a[:, :h] + a[:, h:2 * h]
        s = np.zeros(nx)
        for warp in a[:, 0]:
            s = s + warp
        return s * inv2

    d = np.zeros_like(v)
    for m in range(lo, hi + 1):
        c, s = cos[m], sin[m]
        d = d + (coef(c) * c[:, None].astype(np.float64) + coef(s) * s[:, None].astype(np.float64))
    return v - d


@pytest.mark.parametrize("nz,nx,text", CASES)
def test_bands_bit_for_bit(cuda, orc, nz, nx, text):
    from kh_simulations_b200 import _lib
    from kh_simulations_b200._lib import Grid
    from kh_simulations_b200.config import derive, loads, step_params
    from kh_simulations_b200.run import KHRun

    base = BASE + f"nz_override = {nz}\nnx_override = {nx}\n"
    cfg = loads(base + text, "bands")
    d = derive(cfg)
    run = KHRun(cfg)
    run.init()
    run.add_noise(1e-3, seed=6)
    s0 = run.state_numpy().copy()
    run.step(1)
    s1 = run.state_numpy().copy()
    n0 = _lib.launch_count()
    run.step(1)
    assert _lib.launch_count() - n0 == 2 + cfg.suppress_kz0 + 2 * len(d.bands)  # the separate kernels
    s2 = run.state_numpy()
    run.close()
    mhi = max(hi for _, hi in d.bands)
    c, sn = np.empty((mhi + 1, nz), np.float32), np.empty((mhi + 1, nz), np.float32)
    _lib.check(_lib.load().ymkh_twiddles(nz, 0, mhi, c.ctypes.data_as(C.c_void_p), sn.ctypes.data_as(C.c_void_p)), "tw")
    if nz % 32 == 0:
        want = orc.step(Grid(nx, nz, d.dx, d.dz), step_params(cfg, d), s0.copy(), 2, twiddles=(c, sn))
        assert np.array_equal(s2.view(np.uint64), want.view(np.uint64))
        return
    plain = KHRun(loads(base, "plain"))  # the step without its bands, then those
    for before, after in ((s0, s1), (s1, s2)):
        plain.set_state(before)
        plain.step(1)
        want = plain.state_numpy().copy()
        for a in FILTERED:
            for lo, hi in d.bands:
                want[a] = _subtract_band(want[a], lo, hi, c, sn)
        assert np.array_equal(after.view(np.uint64), want.view(np.uint64))
    plain.close()
