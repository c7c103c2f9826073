"""The tuner's candidates (no GPU needed)."""
import pytest

from kh_simulations_b200 import autotune


@pytest.mark.parametrize("nx,nz", [(64, 512), (96, 128), (100, 4096), (128, 64), (768, 256), (8, 32)])
def test_candidates_hold_the_form_that_a_run_takes_by_itself(nx, nz):
    """Else tuning replaces the default by a narrower strip, faster or not."""
    shapes = autotune.candidates(nx, nz)
    assert (32, 1) in shapes and (128, 1) in shapes
    assert len(set(shapes)) == len(shapes)
