"""The bits of a row-major product depend on the graph, the width and the values
alone: the vector form, the padded copy and the element-wise form (few entries a
row) agree bit for bit, whatever the alignment and strides of X and Y, on a first
call, on a later one, and on a call that a capture makes before any other."""
import numpy as np
import pytest
import torch

from gpu_util import TOL_F32, dense_x, fp64_reference, rel
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F, B = torch.float32, torch.bfloat16


def coo(n, per_row, seed):
    rng = np.random.Generator(np.random.Philox(seed))
    m = int(n * per_row)
    row = rng.integers(0, n, m).astype(np.int32)
    row[:m // 8] = 5  # a hub row
    return row, rng.integers(0, n, m).astype(np.int32), rng.standard_normal(m).astype(np.float32)


def build(n, c):
    return S.Graph.from_coo_device(n, *[torch.from_numpy(a).to(DEV) for a in c], nparts=2)


def place(x, stride, off):
    """x as a view with this row stride, its first element `off` elements in."""
    n, K = x.shape
    flat = torch.full((n * stride + off,), float("nan"), device=DEV, dtype=x.dtype)
    v = flat[off:off + n * stride].view(n, stride)[:, :K]
    v.copy_(x)
    return v


@pytest.mark.parametrize("per_row", [1.5, 6, 20])
@pytest.mark.parametrize("xdt,ydt", [(F, F), (F, B), (B, F), (B, B)])
@pytest.mark.parametrize("K", [1, 3, 8, 13, 16, 33, 64, 100, 128, 136, 257, 264, 520])
def test_same_bits(per_row, xdt, ydt, K):
    n = 1501
    c = coo(n, per_row, seed=K)
    x = torch.from_numpy(dense_x(n, K, seed=K)).to(DEV).to(xdt)
    ld = (K + 7) // 8 * 8
    g = build(n, c)
    want = g.spmm(place(x, ld, 0), place(torch.zeros((n, K), device=DEV, dtype=ydt), ld, 0)).clone()
    tol = TOL_F32 if ydt == F else 4e-3
    assert rel(want.float().cpu().numpy(), fp64_reference(n, *c, x.float().cpu().numpy())) <= tol
    for stride, off in ((K, 0), (K + 1, 1), (ld, 3), (ld + 8, 8)):
        X = place(x, stride, off)
        for yo in (0, 1):
            Y = place(torch.zeros((n, K), device=DEV, dtype=ydt), stride, yo)
            g.spmm(X, Y)
            assert torch.equal(Y, want), (stride, off, yo)
    fresh = build(n, c)
    X, Y = place(x, K + 1, 1), torch.zeros((n, K), device=DEV, dtype=ydt)
    cg = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cg):
        fresh.spmm(X, Y)
    cg.replay()
    torch.cuda.synchronize()
    assert torch.equal(Y, want)
    del cg
