"""The row-major launches overlap the kernels before them (programmatic dependent
launch): products chained through each other's outputs and through other
kernels, copies and fills, on one stream, on two ordered by events, and captured
in a CUDA graph with each kind of predecessor, equal the same steps one at a
time."""
import pytest
import torch

from gpu_util import graph_case
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def chain(g, x, y, z, sync):
    """z = A (relu(A (2 A x)) + 1), then y += A z, with a fill and copies between."""
    g.spmm(x, y)
    sync()
    y.mul_(2)
    sync()
    z.zero_()
    sync()
    g.spmm(y, z, accumulate=True)
    sync()
    torch.relu_(z)
    sync()
    y.copy_(z)
    sync()
    y.add_(1)
    sync()
    g.spmm(y, z)
    sync()
    g.spmm(z, y, accumulate=True)
    sync()


@pytest.mark.parametrize("scale,K,thr", [(9, 32, 0), (11, 16, 8), (13, 128, 16), (13, 36, 10 ** 6)])
def test_chained_products(scale, K, thr):
    n, row, col, val, ps = graph_case(scale, 12, seed=scale, nparts=2)
    g = S.Graph(ps, hub_threshold=thr)
    x = torch.randn((n, K), device=DEV)
    y, z = torch.zeros_like(x), torch.zeros_like(x)
    chain(g, x, y, z, torch.cuda.synchronize)
    want = (y.clone(), z.clone())
    for rep in range(50):
        chain(g, x, y, z, lambda: None)
    torch.cuda.synchronize()
    assert torch.equal(y, want[0]) and torch.equal(z, want[1])
    cg = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cg):
        chain(g, x, y, z, lambda: None)
    y.fill_(float("nan"))
    for rep in range(20):
        cg.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want[0]) and torch.equal(z, want[1])
    # two streams ordered by events: the product is the first work after the wait
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    big = torch.randn((3000, 3000), device=DEV)
    torch.cuda.synchronize()
    for rep in range(10):
        with torch.cuda.stream(s1):
            big @ big
            x2 = x * 2
            e = s1.record_event()
        s2.wait_event(e)
        with torch.cuda.stream(s2):
            y2 = g.spmm(x2, stream=s2)
            e2 = s2.record_event()
        s1.wait_event(e2)
        x2.record_stream(s2)
        y2.record_stream(s1)
        with torch.cuda.stream(s1):
            g.spmm(y2, z, stream=s1)
    torch.cuda.synchronize()
    y1 = g.spmm(x * 2)
    assert torch.equal(z, g.spmm(y1))
