"""Label widening when no memory is to be had for its threads: it runs on the caller's thread alone and returns, rather
than let an exception out of a C entry point.  C++ allocations are made to fail by a preloaded operator new."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

FAILING_NEW = r"""
#include <cstdlib>
#include <new>
static int left = -1;                      // allocations that still succeed; negative: all
extern "C" void allow_new(int n) { left = n; }
void* operator new(std::size_t n) {
    if (left == 0) throw std::bad_alloc();
    if (left > 0) left--;
    return std::malloc(n ? n : 1);
}
"""

CALL = r"""
import ctypes, sys
import numpy as np
from mcx_gb300._lib import lib
allow = ctypes.CDLL(sys.argv[1]).allow_new
vol = (np.arange(160 * 150 * 140) % 100).astype(np.uint8).reshape(160, 150, 140)
for spare in (0, 1, 2, 3):
    out = np.zeros(vol.size, np.uint32)
    allow(spare)
    rc = lib.mcxg_widen_labels(vol.ctypes.data, 1, 0, *vol.shape, out.ctypes.data)
    allow(-1)
    assert rc == 0 and np.array_equal(out, vol.ravel(order="F")), spare
print("widened")
"""


def test_labels_without_memory_for_threads(built, tmp_path):
    src, so = tmp_path / "new.cpp", tmp_path / "libnew.so"
    src.write_text(FAILING_NEW)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    p = subprocess.run([sys.executable, "-c", CALL, str(so)], cwd=ROOT, capture_output=True, text=True,
                       env={"LD_PRELOAD": str(so), "PATH": "/usr/bin:/bin", "PYTHONPATH": str(ROOT)}, timeout=300)
    assert p.returncode == 0 and "widened" in p.stdout, (p.returncode, p.stdout, p.stderr[-2000:])
