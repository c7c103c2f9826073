"""The column stages as one kernel (sponge, xi_cut, z-mean, band filters,
z-hyperdiffusion for NZ up to 512): every number of 32-row warps it has a
different path for (one, a power of two, three, sixteen), ragged columns
(NX = 40, and 33: a last tile of one column), several bands, bands of fewer
modes than a block, of exactly one and of one more.  Against the oracle, bit
for bit; and, member by member, batches (which take the kernel for every
member) against lone runs whose single stages run separately."""
import ctypes as C

import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

KZ0, HYPER = "suppress_kz0 = 1\n", "hyp_diff = 5e-5\n"
STAGES = {
    "kz0_hyper": KZ0 + HYPER,
    "kz0_band": KZ0 + "kz_bands = 3-10\n",
    "band_hyper": "kz_bands = 2-8\n" + HYPER,
    "nine_modes_kz0": KZ0 + "kz_bands = 2-10\n",
    "three_bands_all": KZ0 + HYPER + "kz_suppress_max = 2\nkz_suppress_hi = 7\nkz_bands = 11-12\n",
    "keep_third_hyper": HYPER + "kz_keep_max = {third}\n",
}


def _config(stages, nz, nx):
    from kh_simulations_b200.config import loads

    return loads(BASE + stages.format(third=nz // 3) + f"nz_override = {nz}\nnx_override = {nx}\n", "col")


def _twiddles(d):
    from kh_simulations_b200 import _lib

    if not d.bands:
        return None
    mhi = max(hi for _, hi in d.bands)
    c, s = np.empty((mhi + 1, d.nz), np.float32), np.empty((mhi + 1, d.nz), np.float32)
    _lib.check(_lib.load().ymkh_twiddles(d.nz, 0, mhi, c.ctypes.data_as(C.c_void_p), s.ctypes.data_as(C.c_void_p)), "tw")
    return c, s


@pytest.mark.parametrize("nz,nx", [(32, 40), (64, 33), (96, 40), (128, 40), (256, 33), (512, 40)])
@pytest.mark.parametrize("stages", sorted(STAGES))
def test_step_vs_oracle(cuda, orc, stages, nz, nx):
    from kh_simulations_b200._lib import Grid
    from kh_simulations_b200.config import derive, step_params
    from kh_simulations_b200.run import KHRun

    if "suppress_kz0" in STAGES[stages] and nz == 96:
        pytest.skip("the z-mean needs a power of two")
    cfg = _config(STAGES[stages], nz, nx)
    d = derive(cfg)
    run = KHRun(cfg)
    run.init()
    run.add_noise(1e-3, seed=4)
    s0 = run.state_numpy().copy()
    run.step(2)
    s = run.state_numpy()
    run.close()
    want = orc.step(Grid(d.nx, d.nz, d.dx, d.dz), step_params(cfg, d), s0.copy(), 2, twiddles=_twiddles(d))
    assert np.array_equal(s.view(np.uint64), want.view(np.uint64))


def test_batch_members_equal_lone_runs(cuda):
    """Single stages: separate kernels alone, the fused one in the batch."""
    from kh_simulations_b200.batch import KHBatch
    from kh_simulations_b200.run import KHRun

    specs = [(KZ0, 64, 96), (KZ0, 256, 40), (KZ0, 512, 64), (HYPER, 32, 40), (HYPER, 96, 64), ("xi_sponge = 4\n", 64, 64),
             ("xi_sponge = 6\nsigma_sponge = 5\nxi_cut = 8\n", 128, 48), ("xi_cut = 7\n", 32, 33), ("kz_keep_max = 85\n", 256, 40),
             ("kz_keep_max = 21\n", 64, 128), (KZ0 + HYPER + "xi_sponge = 5\nkz_suppress_hi = 9\n", 128, 64), ("", 64, 64),
             (KZ0, 1024, 40), ("filter_engine = tf32x3\nkz_keep_max = 42\n", 128, 128)]
    lone, runs = [], []
    for stages, nz, nx in specs:
        for keep in (lone, runs):
            r = KHRun(_config(stages, nz, nx))
            r.init()
            r.add_noise(1e-3, seed=9)
            keep.append(r)
    batch = KHBatch()
    for r in runs:
        batch.add(r)
    batch.step(5)
    batch.check()
    for r, b, spec in zip(lone, runs, specs):
        r.step(5)
        assert np.array_equal(r.state_numpy().view(np.uint64), b.state_numpy().view(np.uint64)), spec
    batch.close()


def test_batch_follows_a_members_new_parameters(cuda):
    """ymkh_set_params on a member between steps: the batch's tables are rebuilt."""
    from kh_simulations_b200 import _lib
    from kh_simulations_b200.batch import KHBatch
    from kh_simulations_b200.config import step_params
    from kh_simulations_b200.run import KHRun

    a, b = _config(KZ0, 64, 64), _config(KZ0 + HYPER + "kz_bands = 3-9\n", 64, 64)
    runs = [KHRun(a) for _ in range(4)]
    ref = KHRun(a)
    for r in runs + [ref]:
        r.init()
        r.add_noise(1e-3, seed=2)
    batch = KHBatch()
    for r in runs:
        batch.add(r)
    batch.step(3)
    ref.step(3)
    p = step_params(b)
    for r in (runs[1], ref):
        _lib.check(r.lib.ymkh_set_params(r.ctx, C.byref(p)), "ymkh_set_params")
    batch.step(6)
    ref.step(6)
    assert np.array_equal(runs[1].state_numpy(), ref.state_numpy())
    assert not np.array_equal(runs[0].state_numpy(), ref.state_numpy())
    batch.close()


@pytest.mark.parametrize("nz,nx", [(64, 130), (128, 96), (1024, 40)])
@pytest.mark.parametrize("bands", ["kz_keep_max = {third}\n", "kz_bands = 3-9,12-20\n"])
def test_zmean_taken_off_by_the_tf32_filter(cuda, nz, nx, bands):
    """suppress_kz0 with the TF32 engine, whose first band takes the z-means
    off, bit for bit the z-mean stage followed by the filter.  On a fluid at
    rest without fields, sweeps and field update leave Az2 and Az3 as they are,
    so the two stages can be had one after the other in two runs."""
    from kh_simulations_b200.run import KHRun

    tf32 = "filter_engine = tf32x3\n" + bands
    runs = [KHRun(_config(s, nz, nx)) for s in (KZ0 + tf32, KZ0, tf32)]
    both, mean, band = runs
    st = np.zeros((24, nz, nx))
    rng = np.random.default_rng(nz + nx)
    st[10:12] = rng.normal(0.3, 1.0, size=(2, nz, nx))
    st[[12, 18]] = 1.0
    st[15], st[21] = 1.0, -1.0
    both.set_state(st)
    mean.set_state(st)
    both.step(1)
    mean.step(1)
    s = mean.state_numpy()
    assert not np.array_equal(s[10:12], st[10:12]) and np.array_equal(s[12:], st[12:])
    band.set_state(s)
    band.step(1)
    a, b = both.state_numpy(), band.state_numpy()
    assert not np.array_equal(a[10:12], s[10:12])
    assert np.array_equal(a[10:12].view(np.uint64), b[10:12].view(np.uint64))
    for r in runs:
        r.close()
