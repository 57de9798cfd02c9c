"""First calls under CUDA-graph capture of products that need no workspace (GPU).

A route that sums its K ranges inside a cluster asks for no workspace, so its
first call on a stream that the library has not seen records cleanly, and the
replay equals a direct call bit for bit.
"""
from __future__ import annotations

import pytest

from gemm_routes import dgemm_route, sgemm_route

pytestmark = pytest.mark.gpu


def _capture(blas, call, out):
    """`call` recorded on a new stream of a freshly started library, replayed into `out`."""
    import torch
    blas.shutdown()  # gives back every stream's workspace
    direct = out.clone()
    call(direct)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        call(out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, direct)


def _operands(m, n, k, dtype):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    make = lambda c, r: torch.rand((c, r), generator=g, device="cuda", dtype=dtype) * 2 - 1  # noqa: E731
    return make(k, m), make(n, k), make(n, m)


@pytest.mark.parametrize("m,n,k", [(256, 256, 256), (1024, 512, 512), (2048, 512, 2048)])
def test_dgemm(blas, m, n, k):
    import torch
    r = dgemm_route(m, n, k)
    assert r.cluster > 1 and r.splits > 1
    a, b, c = _operands(m, n, k, torch.float64)
    _capture(blas, lambda x: blas.dgemm_device("N", "N", m, n, k, 1.5, a, m, b, k, 0.5, x, m), c)


@pytest.mark.parametrize("m,n,k", [(512, 512, 512), (512, 512, 1300)])
def test_sgemm(blas, m, n, k):
    import torch
    r = sgemm_route(m, n, k)
    assert r.cluster and r.splits > 1
    a, b, c = _operands(m, n, k, torch.float32)
    _capture(blas, lambda x: blas.sgemm_device("N", "N", m, n, k, 1.5, a, m, b, k, 0.5, x, m), c)


@pytest.mark.parametrize("n,k", [(300, 200), (700, 600)])
def test_dsyrk(blas, n, k):
    import torch
    r = dgemm_route(n, n, k, tri=1)
    assert r.cluster > 1 and r.splits > 1
    a, _, c = _operands(n, n, k, torch.float64)
    _capture(blas, lambda x: blas.dsyrk_device("U", "N", n, k, 1.5, a, n, 0.5, x, n), c)
