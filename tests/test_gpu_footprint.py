"""server.footprint() counts what a run holds on the device, diagnostics and
z-means included (NX so large that what belongs to columns is in the tens of MiB)."""
import numpy as np
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu

TF32 = "kz_keep_max = 10\nsuppress_kz0 = 1\nfilter_engine = tf32x3\n"


@pytest.mark.parametrize("nz,nx,text", [(32, 1 << 18, TF32), (32, 1 << 18, "kz_keep_max = 14\n"), (4, 1 << 20, ""),
                                        (2048, 2048, "")])
def test_footprint_covers_the_allocations(cuda, nz, nx, text):
    import torch

    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun
    from kh_simulations_b200.server import footprint

    def use(nz, nx):
        r = KHRun(loads(BASE + f"nz_override = {nz}\nnx_override = {nx}\n" + text))
        r.init()
        r.step(1)
        r.energy()
        r.mode_amp()
        r.circ_amp("By", 1, weight=np.ones(nx))
        r.gauss()
        torch.cuda.synchronize()
        return r

    small = use(32, 64)  # loads the kernels
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    big = use(nz, nx)
    used, counted = free - torch.cuda.mem_get_info()[0], footprint(big.cfg)
    slack = 16 << 20  # allocations come in blocks of 2 MiB
    assert counted - slack <= used <= counted + slack, (used, counted)
    small.close()
    big.close()
