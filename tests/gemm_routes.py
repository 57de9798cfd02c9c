"""The planner's routing rules as a Python function (compiled from csrc/planner.cpp, no GPU needed)."""
from __future__ import annotations

import ctypes as C
import functools
import os
import subprocess
import tempfile
from collections import namedtuple
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))

TILE_128x128, TILE_64x64 = 0, 5
TILES, TMA_128, WS_64, CLUSTER_64 = range(4)

Route = namedtuple("Route", "tile splits kernel cluster ranges k_chunk")
SgemmRoute = namedtuple("SgemmRoute", "splits cluster halves")


@functools.lru_cache(maxsize=None)
def _shim():
    with tempfile.TemporaryDirectory() as tmp:
        so = Path(tmp) / "route_shim.so"
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CUDA / 'include'}",
                        f"-I{ROOT / 'zynum_b200' / 'csrc'}", str(ROOT / "tests" / "cpp" / "route_shim.cpp"),
                        str(ROOT / "zynum_b200" / "csrc" / "planner.cpp"), "-o", str(so)], check=True)
        return C.CDLL(str(so))


def dgemm_route(m, n, k, tri=0, tma=True, automatic=True, sms=148):
    out = (C.c_int * 6)()
    _shim().dgemm_route(m, n, k, tri, int(tma), int(automatic), sms, out)
    return Route(*out)


def sgemm_route(m, n, k, sms=148):
    out = (C.c_int * 3)()
    _shim().sgemm_route(m, n, k, sms, out)
    return SgemmRoute(*out)
