"""The diagnostics at the edges of their partitions: one 32-column tile and one
column more, row ranges shorter and longer than a 64-row phase tile, cells per
thread of one and of several, grids of a few cells.  Against numpy at 64 bits,
with the tolerances of the small-grid tests (compensated or pairwise sums on
both sides)."""
import numpy as np
import pytest

from cases import BASE
from oracle import diagnostics as od

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx", [(4, 4), (8, 33), (70, 32), (129, 96), (2048, 5), (33, 4099), (700, 1500)])
def test_diagnostics_vs_numpy(cuda, nz, nx):
    import torch

    from kh_simulations_b200 import growth
    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    run = KHRun(loads(BASE + f"nz_override = {nz}\nnx_override = {nx}\n", "diag"))
    run.init()
    g = torch.Generator(device="cuda").manual_seed(nz * 10007 + nx)
    st = run.state
    st += 0.01 * torch.randn(st.shape, dtype=torch.float64, device="cuda", generator=g)
    s = run.state_numpy()

    n = np.maximum(s[[12, 18]], 1e-10)
    cell = 0.5 * (s[0:9] ** 2).sum(axis=0) + (0.5 * (s[[13, 19]] ** 2 + s[[14, 20]] ** 2) / n).sum(axis=0)
    assert run.energy() == pytest.approx(float(cell.sum()), rel=1e-13)

    for weight in (None, growth.xi_weight(nx, run.d.dx, eps=run.d.eps, lx=run.d.lx)):
        for k in (0, 1, min(3, nz // 2)):
            re, im = s[od.IDX["By2"]], s[od.IDX["By3"]]
            col = (np.abs(re).sum(axis=0) + np.abs(im).sum(axis=0)) / nz
            scale = float(col.mean() if weight is None else np.dot(col, weight))
            got = run.circ_amp("By", k=k, weight=weight)
            for a, b in zip(got, od.circ_amp(re, im, k, weight)):
                assert abs(a - b) <= 1e-12 * abs(b) + 1e-13 * scale, (k, a, b)

    ref = od.gauss_terms(s, run.d.dx, run.d.dz, run.d.alpha)
    q = run.gauss()
    got = np.concatenate([q["G"], q["div_E"], q["nonabelian"], q["rho"], q["lhs"], [(q["Etot_scale"] - 1e-30) * run.d.dx]])
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=0)
    run.close()
