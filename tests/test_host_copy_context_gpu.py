"""Staged transfers of the host entry points from a CUDA context of the caller's own (GPU)."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

CODE = r"""
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
cu = C.CDLL("libcuda.so.1")
dev, ctx, cur, flags, active = C.c_int(), C.c_void_p(), C.c_void_p(), C.c_uint(), C.c_int()
assert cu.cuInit(0) == 0 and cu.cuDeviceGet(C.byref(dev), 0) == 0
assert cu.cuCtxCreate_v2(C.byref(ctx), 0, dev) == 0
from zynum_b200 import blas
rng = np.random.default_rng(1)
for beta in (0.0, 0.5):
    m, n, k = 1100, 1200, 1000  # 8 MB and more each: staged
    a, b, c = (np.asfortranarray(rng.uniform(-1, 1, s)) for s in ((m, k), (k, n), (m, n)))
    ref = a @ b + beta * c
    bound = 5 * k * 2.0 ** -53 * (np.abs(a) @ np.abs(b) + np.abs(c))
    blas.dgemm("N", "N", m, n, k, 1.0, a, m, b, k, beta, c, m)
    assert np.all(np.abs(c - ref) <= bound)
assert cu.cuCtxGetCurrent(C.byref(cur)) == 0 and cur.value == ctx.value
assert cu.cuDevicePrimaryCtxGetState(dev, C.byref(flags), C.byref(active)) == 0
assert active.value == 0, "a copying thread brought up the device's primary context"
"""


def test_copies_run_in_the_callers_context():
    r = subprocess.run([sys.executable, "-c", CODE, str(ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and not r.stderr, r.stderr
