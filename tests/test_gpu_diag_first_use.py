"""A run's first energy and amplitude take no device memory that the run does
not already hold: the server and campaigns fill the memory with states."""
import pytest

from cases import BASE

pytestmark = pytest.mark.gpu


def test_first_energy_and_amplitude_allocate_nothing(cuda):
    import torch

    from kh_simulations_b200.config import loads
    from kh_simulations_b200.run import KHRun

    def run(nz, nx):
        r = KHRun(loads(BASE + f"nz_override = {nz}\nnx_override = {nx}\n"))
        r.init()
        return r

    small = run(32, 48)  # loads the kernels
    want = small.energy(), small.mode_amp(k=1)
    big = run(4, 1 << 18)  # amplitude sums of 8 MiB
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    big.energy()
    big.mode_amp(k=1)
    assert torch.cuda.mem_get_info()[0] == free
    assert (small.energy(), small.mode_amp(k=1)) == want
    small.close()
    big.close()
