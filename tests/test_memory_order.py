"""Orderings that the kernels owe to the memory model and that no run shows
when they are missing, checked in the source (no GPU needed).

* Shared memory that ordinary stores or cp.async have written is handed to TMA
  only behind ``fence.proxy.async``: a barrier orders the threads, not the two
  proxies.
* A kernel that starts before its predecessor ends reads what that one writes
  through plain pointers: ``const __restrict__`` data may be read before the
  ``griddepcontrol.wait``.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "kh_simulations_b200" / "csrc"


def _code(name):
    """The source without comments, white space collapsed."""
    text = re.sub(r"/\*.*?\*/", " ", (CSRC / name).read_text(), flags=re.S)
    return re.sub(r"\s+", " ", re.sub(r"//[^\n]*", " ", text))


@pytest.mark.parametrize("name,pieces", [("ymkh_fct.cu", 2), ("ymkh_maxwell.cu", 1)])
def test_copied_piece_is_fenced_before_tma_may_take_its_slots(name, pieces):
    """A piece of rows copied with cp.async can be followed by one copied by
    TMA into the same slots (a batch of wall and periodic runs): every thread
    that copied ends the piece with its copies done and the fence."""
    ends = re.findall(r"if \(!bulk\) \{? ?cp_async_wait<0>\(\);(.{0,44})", _code(name))
    assert len(ends) == pieces
    for after in ends:
        assert after.startswith(" if (T.nruns > 1) fence_proxy_async(); }"), after  # a run keeps to one kind of copy


def test_patched_columns_are_fenced_before_tma_retakes_the_slot():
    """The wrapped columns of an edge strip are stored into the row's slots,
    which TMA overwrites some rows later: stores, fence, barrier."""
    code = _code("ymkh_fct.cu")
    body = re.search(r"auto patch_row = \[&\]\(.*?\) \{(.*?)\} ;|auto patch_row = \[&\]\(.*?\) \{(.*?)\};", code)
    assert re.search(r"= src\[e\]; \} fence_proxy_async\(\); $", body.group(1) or body.group(2))
    assert re.search(r"if \(patch\) \{ patch_row\([^;]*\); coef_bar\(\); \}", code)


def test_dependent_kernels_read_partial_sums_through_plain_pointers():
    code = _code("ymkh_diag.cu")
    kernels = re.findall(r"__global__ void __launch_bounds__\(\w+\) (\w+)\(([^)]*)\) \{ dependency_wait\(\);", code)
    assert sorted(k for k, _ in kernels) == ["energy_final_kernel", "gauss_final_kernel", "mode_amp_final_kernel"]
    assert {k for k, _ in kernels} == set(re.findall(r"launch_dependent\((\w+_kernel)", code))
    for _, params in kernels:
        part = params.split(",")[0]
        assert part.endswith(" part") and "const" not in part and "__restrict__" not in part, part
