"""Which runs take the one column kernel, and which members of a batch share it:
kernels launched a step on both sides of each line of the rules, and every
member bit for bit as alone either way."""
import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

KZ0, HYPER = "suppress_kz0 = 1\n", "hyp_diff = 5e-5\n"


def _bands(modes):
    return f"kz_suppress_hi = {modes + 1}\n"  # modes 2 .. modes + 1


# four members; launches a step besides the FCT and Maxwell: 1 shared, or 4 x the member's own
CASES = [
    (160, 512, _bands(10), 1),
    (160, 512, _bands(11), 8),
    (160, 256, _bands(24), 1),
    (160, 256, _bands(25), 8),
    (160, 64, _bands(48), 1),
    (160, 64, _bands(49), 8),
    (128, 512, _bands(40), 1),
    (64, 512, KZ0, 1),
    (128, 480, KZ0, 1),
    (128, 512, KZ0, 4),
    (128, 512, KZ0 + HYPER, 1),
    (256, 128, KZ0 + _bands(49), 1),
    (288, 128, HYPER + _bands(49), 12),
    (512, 64, KZ0 + _bands(49), 1),
    (512, 128, KZ0 + _bands(48), 1),
    (512, 128, KZ0 + HYPER + _bands(49), 1),
]
# a lone run: one kernel, or its own
ALONE = [
    (512, 192, KZ0 + _bands(49), 1),   # 108 CTAs with work
    (512, 40, KZ0 + _bands(49), 3),    # 36
    (512, 256, HYPER + _bands(49), 3),  # 168: a second turn nearly empty
    (512, 256, HYPER + _bands(48), 1),
    (288, 192, HYPER + _bands(49), 1),
    (256, 40, KZ0 + _bands(49), 1),
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


@pytest.mark.parametrize("nz,nx,text,launches", ALONE)
def test_column_kernel_of_a_lone_run(cuda, orc, nz, nx, text, launches):
    import ctypes as C

    from kh_simulations_b200 import _lib
    from kh_simulations_b200._lib import Grid
    from kh_simulations_b200.config import derive, loads, step_params
    from kh_simulations_b200.run import KHRun

    cfg = loads(BASE + f"nz_override = {nz}\nnx_override = {nx}\n" + text)
    d = derive(cfg)
    r = KHRun(cfg, graph_steps=0)
    r.init()
    s0 = r.state_numpy().copy()
    n0 = _lib.launch_count()
    r.step(1)
    assert _lib.launch_count() - n0 == 2 + launches
    s = r.state_numpy()
    r.close()
    mhi = max(hi for _, hi in d.bands)
    c, sn = np.empty((mhi + 1, nz), np.float32), np.empty((mhi + 1, nz), np.float32)
    _lib.check(_lib.load().ymkh_twiddles(nz, 0, mhi, c.ctypes.data_as(C.c_void_p), sn.ctypes.data_as(C.c_void_p)), "tw")
    want = orc.step(Grid(nx, nz, d.dx, d.dz), step_params(cfg, d), s0.copy(), 1, twiddles=(c, sn))
    assert np.array_equal(s.view(np.uint64), want.view(np.uint64))
