"""The 128-wide FCT form (one warp per swept variable) at the sizes where it
can go wrong, bit for bit against the split FCT form, whose kernels share none
of its staging: grids at the edges of its 120-column strips and of its 128-wide
TMA boxes, wrapped columns in the first and the last strip, rows copied array
by array (NX below 128, arrays not evenly spaced), element by element (walls,
odd NX), with and without warm_T; segments that make a piece one row or the
whole column; rows with infinities, NaNs and huge values, where the limiter
leaves its finite form; and a batch that mixes all of these."""
import ctypes as C

import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

WALL = BASE.replace("run_mode = 6", "run_mode = 0")
GRIDS = {  # name: (ini, NZ, NX)
    "one_box": (BASE, 7, 128),
    "two_strips": (BASE, 33, 240),
    "last_strip_of_two_columns": (BASE, 20, 242),
    "wrap_inside_last_box": (BASE, 16, 364),
    "below_box": (BASE, 64, 124),
    "narrow": (BASE, 40, 24),
    "odd": (BASE, 27, 131),
    "wall_even": (WALL, 24, 250),
    "wall_odd": (WALL, 31, 121),
    "warm": (BASE + "warm_T = 0.01\n", 24, 368),
    "warm_wall": (WALL + "warm_T = 0.01\n", 18, 130),
}


def _run(name):
    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    ini, nz, nx = GRIDS[name]
    run = KHRun(loads(ini + f"nz_override = {nz}\nnx_override = {nx}\n", name))
    run.init()
    run.add_noise(1e-3, seed=11)
    return run


def _form(run, mode, seg=1):
    from kh_simulations_b200 import _lib

    _lib.check(run.lib.ymkh_set_fct_mode(run.ctx, mode), "ymkh_set_fct_mode")
    _lib.check(run.lib.ymkh_set_fct_shape(run.ctx, 128, seg), "ymkh_set_fct_shape")


def _states(run, st, shapes, steps):
    from kh_simulations_b200 import _lib

    out = []
    for mode, seg in shapes:
        _form(run, mode, seg)
        run.set_state(st)
        run.step(steps)
        out.append(run.state_numpy().copy())
        _lib.check(run.lib.ymkh_check(run.ctx, None), "ymkh_check")
    return out


@pytest.mark.parametrize("name", sorted(GRIDS))
def test_strip_form_matches_split(cuda, name):
    from kh_simulations_b200 import _lib

    run = _run(name)
    st = run.state_numpy().copy()
    split, *strips = _states(run, st, [(_lib.FCT_SPLIT, 1), (_lib.FCT_FUSED, 1), (_lib.FCT_FUSED, 5),
                                       (_lib.FCT_FUSED, run.d.nz)], 3)
    assert np.isfinite(split).all()
    for s in strips:
        assert np.array_equal(split.view(np.uint64), s.view(np.uint64))
    run.close()


@pytest.mark.parametrize("value", [np.inf, np.nan, 1e200, -1e300, 1e-310])
@pytest.mark.parametrize("name", ["two_strips", "wall_odd"])
def test_strip_form_with_non_finite_rows(cuda, name, value):
    """One cell of a fluid and of a field array holds the value: the rows it
    reaches take the NaN-exact limiter, and every cell agrees with the split
    form (NaNs by position)."""
    from kh_simulations_b200 import _lib

    run = _run(name)
    st = run.state_numpy().copy()
    nz, nx = run.d.nz, run.d.nx
    for k, arr in enumerate((1, 7, 12, 14, 20, 23)):  # Ex2, By2, n A, pz A, pz B, Q3 B
        s = st.copy()
        s[arr, (5 * k + 3) % nz, (37 * k + 2) % nx] = value
        a, b = _states(run, s, [(_lib.FCT_SPLIT, 1), (_lib.FCT_FUSED, 1)], 2)
        assert np.array_equal(a, b, equal_nan=True), (arr, value)
    run.close()


def test_strip_form_with_spaced_arrays(cuda):
    """Arrays bound with different gaps between them: no TMA boxes, one row
    copy per array; the same state as the evenly spaced one."""
    import torch

    from kh_simulations_b200 import _lib

    run = _run("two_strips")
    st = run.state_numpy().copy()
    want, = _states(run, st, [(_lib.FCT_FUSED, 1)], 2)
    n = run.d.nz * run.d.nx
    bufs, ptrs = [], []
    for k in range(2):
        arrs = [torch.empty(n + 2 * i, dtype=torch.float64, device=run.device)[2 * i:] for i in range(24)]
        bufs.append(arrs)
        ptrs.append((C.c_void_p * 24)(*[a.data_ptr() for a in arrs]))
    for i in range(24):
        bufs[0][i].copy_(torch.from_numpy(st[i].reshape(-1)))
    _lib.check(run.lib.ymkh_bind_state2(run.ctx, *ptrs), "ymkh_bind_state2")
    run.step(2)
    torch.cuda.synchronize()
    got = np.stack([a.cpu().numpy().reshape(st.shape[1:]) for a in bufs[run.current]])
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
    run.close()


def test_strip_form_in_a_mixed_batch(cuda):
    from kh_simulations_b200 import _lib
    from kh_simulations_b200.batch import KHBatch

    names = sorted(GRIDS)
    want = []
    for nm in names:
        run = _run(nm)
        want += _states(run, run.state_numpy().copy(), [(_lib.FCT_SPLIT, 1)], 5)
        run.close()
    runs = [_run(nm) for nm in names]
    batch = KHBatch()
    for r in runs:
        batch.add(r)
    batch.step(5)
    batch.check()
    for r, w, nm in zip(runs, want, names):
        assert np.array_equal(r.state_numpy().view(np.uint64), w.view(np.uint64)), nm
    batch.close()


@pytest.fixture(scope="module")
def velocity_checker(cuda, tmp_path_factory):
    import subprocess
    from pathlib import Path

    root = Path(__file__).resolve().parents[1]
    out = tmp_path_factory.mktemp("velcheck") / "libvelcheck.so"
    subprocess.run(["nvcc", "-std=c++17", "-O3", "-fmad=false", "-gencode", "arch=compute_100a,code=sm_100a", "-shared",
                    "-Xcompiler", "-fPIC", f"-I{root / 'include'}", f"-I{root / 'kh_simulations_b200' / 'csrc'}",
                    str(root / "tests" / "kernels" / "velocities_check.cu"), "-o", str(out)],
                   check=True, capture_output=True, timeout=300)
    lib = C.CDLL(str(out))
    lib.velocities_check.argtypes = [C.c_ulonglong, C.c_longlong, C.c_int, C.POINTER(C.c_ulonglong), C.POINTER(C.c_double)]
    return lib


@pytest.mark.parametrize("kind", range(6))
def test_velocities_are_the_ieee_quotients(velocity_checker, kind):
    bad, first = C.c_ulonglong(), (C.c_double * 2)()
    assert velocity_checker.velocities_check(99 + kind, 1 << 28, kind, C.byref(bad), first) == 0
    assert bad.value == 0, (kind, bad.value, first[0], first[1])
