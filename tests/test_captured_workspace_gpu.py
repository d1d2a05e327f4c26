"""A captured product keeps the workspaces it was captured with: replays are right,
and write nowhere else, after wider calls have grown the graph's workspaces and
other graphs have been built in freed memory; a capture that has to size a
workspace itself works too."""
import numpy as np
import pytest
import torch

from gpu_util import TOL_F32, dense_x, fp64_reference, graph_case, rel
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def others(n, m, count):
    """Graphs built on the device into whatever memory is free, and their products."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(7)
    x = torch.randn((n, 32), generator=gen, device=DEV)
    gs = []
    for _ in range(count):
        r, c = (torch.randint(0, n, (m,), generator=gen, device=DEV, dtype=torch.int32) for _ in range(2))
        gs.append(S.Graph.from_coo_device(n, r, c, torch.rand(m, generator=gen, device=DEV)))
    return gs, x, [g.spmm(x) for g in gs]


def capture(g, X, Y, schedule):
    cg = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cg):
        g.spmm(X, Y, schedule=schedule)
    return cg


# hub threshold 48: hub partials as well; 10^6: no hub rows
@pytest.mark.parametrize("K,wider,thr,schedule,ydt", [
    (33, 65, 10 ** 6, S.SCHEDULE_ROWS, torch.float32), (33, 301, 48, S.SCHEDULE_ROWS, torch.float32),
    (32, 512, 48, S.SCHEDULE_ROWS, torch.float32), (32, 256, 48, S.SCHEDULE_FUSED, torch.bfloat16),
    (32, 256, 48, S.SCHEDULE_BUFFER, torch.float32)])
@pytest.mark.parametrize("warm", [True, False])
def test_replay_after_growth(K, wider, thr, schedule, ydt, warm):
    n, row, col, val, ps = graph_case(13, 32, seed=5, nparts=2)  # dense enough for padded copies of X
    g = S.Graph(ps, hub_threshold=thr)
    X = torch.from_numpy(dense_x(n, K, seed=1)).to(DEV)
    ref = fp64_reference(n, row, col, val, X.cpu().numpy())
    tol = TOL_F32 if ydt == torch.float32 else 4e-3  # one rounding to BF16 of each value
    Y = torch.zeros((n, K), dtype=ydt, device=DEV)
    if warm:
        g.spmm(X, Y, schedule=schedule)
    cg = capture(g, X, Y, schedule)
    held = g.get_info().device_bytes
    wide = torch.from_numpy(dense_x(n, wider, seed=2)).to(DEV)
    Yw = torch.zeros((n, wider), dtype=ydt, device=DEV)
    for rep in range(2):
        g.spmm(wide, Yw, schedule=schedule)
    gs, x, want = others(n, 200000, 4)
    for rep in range(2):
        Y.fill_(float("nan"))
        cg.replay()
    torch.cuda.synchronize()
    assert rel(Y.float().cpu().numpy(), ref) <= tol
    assert all(torch.equal(o.spmm(x), w) for o, w in zip(gs, want))
    assert rel(Yw.float().cpu().numpy(), fp64_reference(n, row, col, val, wide.cpu().numpy())) <= tol
    # the captured call's block and the wider one are both counted
    assert g.get_info().device_bytes > held
    del cg
