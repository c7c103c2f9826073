"""A NaN or an infinity in one cell reaches every diagnostic that reads the
cell, and none that does not: the first and last cell of the grid, and one in
the middle of a row range."""
import math

import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu


def _all(r):
    g = r.gauss()
    return {"energy": [r.energy()], "By": r.circ_amp("By", 1), "weighted": r.circ_amp("By", 1, weight=np.ones(r.d.nx)),
            "Az": r.circ_amp("Az", 1), **{k: g[k] for k in ("G", "div_E", "nonabelian", "rho", "lhs")},
            "scale": [g["Etot_scale"]]}


@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("z,x", [(0, 0), (129, 70), (69, 33)])
def test_nonfinite_cell_reaches_the_diagnostics(cuda, bad, z, x):
    import torch

    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    r = KHRun(loads(BASE + "nz_override = 130\nnx_override = 71\n"))
    r.init()
    r.add_noise(1e-3, seed=2)
    st = r.state
    clean = _all(r)
    assert all(np.isfinite(v).all() for v in clean.values())
    readers = {"By2": {"energy", "By", "weighted"}, "Az3": {"Az", "G", "nonabelian", "lhs"},
               "Ex1": {"energy", "G", "div_E", "lhs", "scale"}, "QA1": {"G", "rho"}}
    index = {"By2": 7, "Az3": 11, "Ex1": 0, "QA1": 15}
    for name, hit in readers.items():
        keep = st[index[name], z, x].clone()
        st[index[name], z, x] = bad
        torch.cuda.synchronize()
        for what, v in _all(r).items():
            if what in hit:
                assert not np.isfinite(v).all(), (name, what, v)
            else:
                assert np.array_equal(v, clean[what]), (name, what, v)
        st[index[name], z, x] = keep
    r.close()
