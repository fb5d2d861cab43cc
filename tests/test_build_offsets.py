"""Sequence offsets that descend are refused by both builders before any code is read."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CALL = """
import ctypes as C, sys
import numpy as np
from haystackfm_b200 import _lib as L
codes = np.ones(64, np.uint8)
off = np.array(%s, np.uint64)
opts = L.HfmBuildOpts(32, 0, 1, 0, 1)
out, n = L.u8p(), C.c_size_t()
args = [L.ptr(codes, L.u8p), L.ptr(off, L.u64p), len(off) - 1, None, C.byref(opts), 1]
rc = L.lib().hfm_build_index_gpu(*args, 0, C.byref(out), C.byref(n)) if %r else L.lib().hfm_build_index(*args, C.byref(out), C.byref(n))
print("status", rc)
"""


@pytest.mark.parametrize("gpu", [False, True])
@pytest.mark.parametrize("off", [[0, 10, 5, 20], [0, 64, 1], [20, 0, 64]])
def test_descending_offsets_refused(gpu, off):
    # in a process of its own: a length that wraps would read far past the codes
    r = subprocess.run([sys.executable, "-c", CALL % (off, gpu)], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    assert "status -4" in r.stdout                       # HFM_E_ARG
