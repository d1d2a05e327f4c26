"""Widths and alignments that no vector divides (the row-major schedule copies X
with padded rows and writes Y element by element; below 2 entries a row, and
while a stream is captured without a workspace, the scalar kernel runs):
against FP64, other columns of a wider Y untouched, BF16 outputs the rounded
FP32 ones."""
import numpy as np
import pytest
import torch

from gpu_util import TOL_F32, dense_x, fp64_reference, graph_case, rel
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F, B = torch.float32, torch.bfloat16


@pytest.fixture(scope="module")
def dense_graph():
    n, row, col, val, ps = graph_case(11, 12, seed=3, nparts=3)
    return n, row, col, val, S.Graph(ps, hub_threshold=48, hub_segment=5)


@pytest.fixture(scope="module")
def sparse_graph():
    rng = np.random.Generator(np.random.Philox(9))
    n, m = 3000, 4000  # under 2 entries a row
    row, col = (rng.integers(0, n, m).astype(np.int32) for _ in range(2))
    val = rng.standard_normal(m).astype(np.float32)
    t = [torch.from_numpy(a).to(DEV) for a in (row, col, val)]
    return n, row, col, val, S.Graph.from_coo_device(n, *t, nparts=2)


def check(case, K, xdt, ydt, xpad, xoff, ypad, yoff):
    n, row, col, val, g = case
    Xh = dense_x(n, K, seed=K)
    flat = torch.full((n * (K + xpad) + xoff,), float("nan"), device=DEV).to(xdt)
    X = flat[xoff:].view(n, K + xpad)[:, :K]
    X.copy_(torch.from_numpy(Xh))
    ref = fp64_reference(n, row, col, val, X.float().cpu().numpy())

    def out(dt):
        y = torch.full((n * (K + ypad) + yoff,), 7.0, device=DEV).to(dt)
        return y, y[yoff:].view(n, K + ypad)
    yf, y = out(ydt)
    g.spmm(X, y[:, :K])
    y32f, y32 = out(F)
    g.spmm(X, y32[:, :K])
    assert rel(y32[:, :K].cpu().numpy(), ref) <= TOL_F32
    assert torch.equal(y[:, :K], y32[:, :K].to(ydt))
    for f, v in ((yf, y), (y32f, y32)):
        assert torch.all(v[:, K:] == 7.0) and torch.all(f[:yoff] == 7.0)
    acc = y32.clone()
    g.spmm(X, acc[:, :K], accumulate=True)
    # one rounding of the sum of two equal numbers: exact
    assert torch.equal(acc[:, :K], 2 * y32[:, :K]) and torch.all(acc[:, K:] == 7.0)


@pytest.mark.parametrize("xdt,ydt", [(F, F), (F, B), (B, B), (B, F)])
@pytest.mark.parametrize("K", [1, 2, 3, 5, 7, 9, 15, 17, 31, 33, 63, 65, 74, 127, 129, 257, 301])
def test_odd_widths(dense_graph, K, xdt, ydt):
    check(dense_graph, K, xdt, ydt, 0, 0, 0, 0)


@pytest.mark.parametrize("xdt,ydt", [(F, F), (B, B)])
@pytest.mark.parametrize("K", [3, 32, 36, 128])
@pytest.mark.parametrize("xpad,xoff,ypad,yoff", [(1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 3, 0), (0, 0, 0, 1), (5, 3, 7, 5),
                                                 (8, 8, 8, 8)])
def test_strides_and_alignment(dense_graph, K, xdt, ydt, xpad, xoff, ypad, yoff):
    check(dense_graph, K, xdt, ydt, xpad, xoff, ypad, yoff)


@pytest.mark.parametrize("K", [3, 33, 130])
def test_few_entries_a_row(sparse_graph, K):
    check(sparse_graph, K, F, F, 0, 0, 0, 0)


def test_captured_without_workspace():
    n, row, col, val, ps = graph_case(10, 8, seed=4, nparts=2)
    g = S.Graph(ps, hub_threshold=10 ** 6)  # no hubs: the call allocates nothing when it need not
    X = torch.from_numpy(dense_x(n, 33, seed=1)).to(DEV)
    Y = torch.zeros((n, 33), device=DEV)
    cg = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cg):
        g.spmm(X, Y)
    Y.fill_(float("nan"))
    cg.replay()
    torch.cuda.synchronize()
    assert rel(Y.cpu().numpy(), fp64_reference(n, row, col, val, X.cpu().numpy())) <= TOL_F32
