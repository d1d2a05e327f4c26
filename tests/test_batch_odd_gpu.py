"""Graphs of a batch whose widths or alignments no vector divides: bind sizes all
they need (a run or capture allocates nothing, whatever the graphs ran before),
results are the bits of the graph's own product, and the batch and the graphs'
own calls may run at the same time."""
import numpy as np
import pytest
import torch

from gpu_util import TOL_F32, dense_x, fp64_reference, graph_case, rel
from cola_b200 import spmm as S
from cola_b200.batch import Batch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F, B = torch.float32, torch.bfloat16
KS = [33, 64, 5, 130, 301]


@pytest.fixture(scope="module")
def cases():
    return [graph_case(s, d, seed=s + d, nparts=2) for s, d in ((11, 40), (10, 24), (12, 3), (11, 24), (10, 40))]


def setup(cases, xdt, ydt):
    gs = [S.Graph(c[4], hub_threshold=32, hub_segment=16) for c in cases]
    Xs = [torch.from_numpy(dense_x(c[0], K, seed=K)).to(DEV).to(xdt) for c, K in zip(cases, KS)]
    Ys = [torch.zeros((c[0], K), device=DEV, dtype=ydt) for c, K in zip(cases, KS)]
    return gs, Xs, Ys


def held(gs):
    return [g.get_info().device_bytes for g in gs]


@pytest.mark.parametrize("xdt,ydt", [(F, F), (B, F), (B, B)])
@pytest.mark.parametrize("before", [0, 3, 16])
def test_bind_then_capture(cases, xdt, ydt, before):
    gs, Xs, Ys = setup(cases, xdt, ydt)
    assert all(g.info.hub_rows > 0 for g in gs)
    if before:
        for g, x in zip(gs, Xs):
            g.spmm(x[:, :before].contiguous())
    b = Batch.from_graphs(gs)
    b.bind(Xs, Ys)
    at_bind = held(gs), b.info.device_bytes
    b.capture()
    for rep in range(3):
        [y.fill_(float("nan")) for y in Ys]
        torch.cuda.synchronize()
        b.replay()
    torch.cuda.synchronize()
    captured = [y.clone() for y in Ys]
    [y.fill_(float("nan")) for y in Ys]
    b.run()
    torch.cuda.synchronize()
    assert (held(gs), b.info.device_bytes) == at_bind
    for g, c, x, y, z in zip(gs, cases, Xs, Ys, captured):
        assert torch.equal(y, z)
        alone = torch.empty_like(y)
        g.spmm(x, alone)
        assert torch.equal(y, alone)
        assert rel(y.float().cpu().numpy(), fp64_reference(*c[:4], x.float().cpu().numpy())) <= (
            TOL_F32 if ydt == F else 4e-3)
    # another binding of the same batch
    b.bind([x[:, :-1].contiguous() for x in Xs], [y[:, :-1].contiguous() for y in Ys])
    b.capture()
    b.replay()
    torch.cuda.synchronize()
    b.close()


def test_batch_beside_the_graphs_own_calls(cases):
    gs, Xs, Ys = setup(cases, F, F)
    want = [g.spmm(x).clone() for g, x in zip(gs, Xs)]
    other = [torch.randn((c[0], K), device=DEV) for c, K in zip(cases, KS)]
    want2 = [g.spmm(x).clone() for g, x in zip(gs, other)]
    b = Batch.from_graphs(gs)
    b.bind(Xs, Ys)
    out = [torch.empty_like(y) for y in Ys]
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for rep in range(40):
        for _ in range(3):
            b.run(stream=s1)
            for g, x, y in zip(gs, other, out):
                g.spmm(x, y, stream=s2)
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for y, w in zip(Ys, want))
        assert all(torch.equal(y, w) for y, w in zip(out, want2))
        [y.fill_(float("nan")) for y in Ys + out]
        torch.cuda.synchronize()
    b.close()
