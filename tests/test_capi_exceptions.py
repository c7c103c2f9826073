"""No C++ exception crosses the C boundary: a host allocation that fails inside
an entry point comes back as YMKH_ENOMEM (no GPU needed: the allocation is
the first thing these calls do)."""
import re
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

FAILING_NEW = r"""
#include <cstdlib>
#include <new>
static bool failing = false;
extern "C" void fail_new(int on) { failing = on != 0; }
void* operator new(std::size_t n) {
  if (failing) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void* operator new(std::size_t n, std::align_val_t a) {
  if (failing) throw std::bad_alloc();
  void* p = nullptr;
  if (posix_memalign(&p, static_cast<std::size_t>(a), n ? n : 1) == 0) return p;
  throw std::bad_alloc();
}
"""

CALL = r"""
import ctypes as C, sys
lib, new = C.CDLL(sys.argv[1]), C.CDLL(sys.argv[2])
h = C.c_void_p()
buf = (C.c_int * 512)(256, 256)  # a grid, and parameters that are not reached
new.fail_new(1)
rc = lib.ymkh_batch_create(C.byref(h)) if sys.argv[3] == "batch" else lib.ymkh_create(buf, buf, C.byref(h))
new.fail_new(0)
sys.exit(0 if rc == int(sys.argv[4]) and not h.value else 1)
"""


@pytest.mark.parametrize("what", ["batch", "run"])
def test_failed_host_allocation_is_an_error_code(built, tmp_path, what):
    from kh_simulations_b200 import _lib

    enomem = int(re.search(r"YMKH_ENOMEM = (-\d+)", (ROOT / "include" / "ymkh.h").read_text()).group(1))
    src, so, call = tmp_path / "new.cpp", tmp_path / "new.so", tmp_path / "call.py"
    src.write_text(FAILING_NEW)
    call.write_text(CALL)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-O1", str(src), "-o", str(so)], check=True)
    r = subprocess.run([sys.executable, str(call), str(_lib.LIB_PATH), str(so), what, str(enomem)],
                       env={"LD_PRELOAD": str(so), "PATH": "/usr/bin:/bin"}, capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])


def test_every_entry_point_that_does_work_is_guarded():
    text = (ROOT / "kh_simulations_b200" / "csrc" / "ymkh_capi.cu").read_text()
    body = text[text.index('extern "C" {'):text.index('}  // extern "C"')]
    plain = set(re.findall(r"^(?:int|long long) (ymkh_\w+)\([^;{]*\) \{", body, re.M))
    assert plain == {"ymkh_last_error", "ymkh_launch_count", "ymkh_build_flags", "ymkh_current_buffer",
                     "ymkh_batch_size"}
    assert len(re.findall(r"\) try \{$", body, re.M)) == len(re.findall(r"^\} YMKH_CATCH$", body, re.M)) >= 30
