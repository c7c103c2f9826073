"""ymkh_set_params on a run that is stepping: the tables of its column stages,
and those of a batch that it is in, follow the new bands, also when these
cannot be set up (a band of more modes than a launch can take: the call
fails after the old bands are gone, and the run goes on without any)."""
import copy
import ctypes as C

import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

# the column stages as one kernel, as separate kernels, and on the tensor cores
TEXTS = ["nz_override = 64\nnx_override = 96\nhyp_diff = 5e-5\nkz_suppress_hi = 9\n",
         "nz_override = 256\nnx_override = 64\nkz_suppress_hi = 9\n",
         "nz_override = 64\nnx_override = 128\nkz_keep_max = 21\nsuppress_kz0 = 1\nfilter_engine = tf32x3\n"]


def _run(text):
    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    r = KHRun(loads(BASE + text))
    r.init()
    return r


def _bands(r, *bands):
    """The run's parameters with these extra bands alone."""
    p = copy.copy(r.params)
    p.kz_suppress_max = p.kz_suppress_hi = 0
    p.n_extra_bands = len(bands)
    for i, (lo, hi) in enumerate(bands):
        p.extra_band_lo[i], p.extra_band_hi[i] = lo, hi
    return p


def _set(r, p):
    return r.lib.ymkh_set_params(r.ctx, C.byref(p))


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("text", TEXTS)
def test_bands_that_cannot_be_set_up(cuda, text, batch):
    import torch

    from kh_simulations_b200 import _lib
    from kh_simulations_b200.batch import KHBatch

    r, want = _run(text), _run(text)
    b = KHBatch() if batch else None
    step = b.step if batch else r.step
    if batch:
        b.add(r)
    step(3)
    want.step(3)
    assert _set(r, _bands(r, (2, 70000))) < 0 and "twiddle" in _lib.last_error()
    assert _set(want, _bands(want)) == 0  # no bands
    step(5)
    want.step(5)
    assert np.array_equal(r.state_numpy(), want.state_numpy())
    for q in (r, want):  # and bands again
        assert _set(q, _bands(q, (5, 11), (20, 31))) == 0
    step(5)
    want.step(5)
    torch.cuda.synchronize()
    assert np.array_equal(r.state_numpy(), want.state_numpy())
    if batch:
        b.close()
    r.close()
    want.close()
