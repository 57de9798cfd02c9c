"""Host entry points at the sizes where a transfer changes between threads and a plain copy (GPU).

Two or more pageable transfers of 2 MB take the copying threads, a call's only
one from 8 MB on.  The result must equal the device entry point's on the same
inputs bit for bit, and rows outside C's window must stay untouched.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_host_copy_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,beta", [
    (511, 511, 512, 0.5),    # every transfer just under 2 MB
    (512, 512, 512, 0.5),    # every transfer 2 MB
    (520, 520, 24, 0.5),     # C up and down
    (1023, 1024, 24, 0.0),   # C down only, just under 8 MB
    (1024, 1024, 24, 0.0),   # 8 MB
    (1023, 24, 1024, 0.0),   # A only, just under 8 MB
    (1024, 24, 1024, 0.0),
    (24, 1023, 1024, 0.0),   # B only
    (24, 1024, 1024, 0.0),
])
@pytest.mark.parametrize("pad", [0, 3])
def test_sizes(blas, m, n, k, beta, pad):
    c, c0, dev, dc = _run(blas, "N", "N", m, n, k, pad, beta, 4)
    blas.dgemm_device("N", "N", m, n, k, 1.25, dev["a"], m, dev["b"], k, beta, dc, m)
    assert np.array_equal(c[:, :m], dc.cpu().numpy())
    assert np.array_equal(c[:, m:], c0[:, m:])
