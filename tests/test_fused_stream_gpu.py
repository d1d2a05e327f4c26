"""The streamed form of the fused kernel (BF16 X, and narrow FP32 X, on launches
of many chunks): every lane geometry, chunks that straddle the 32-entry stage
and the warps' spans, all chunk schedules, against FP64 on the features as
stored."""
import pytest
import torch

import cola_b200 as cb
from gpu_util import TOL_F32, dense_x, fp64_reference, rel
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module", params=[(4, 2), (3, 1)])
def graph(request):
    P, gs = request.param
    n, row, col, val = cb.rmat(15, 20, seed=P)
    keep = n - 7  # partitions of uneven size
    m = (row < keep) & (col < keep)
    row, col, val = row[m], col[m], val[m]
    g = S.Graph(cb.PartitionSet.from_coo(keep, row, col, val, P), group_size=gs)
    assert g.info.local_chunks + g.info.remote_chunks >= 148 * 32 * 4  # the streamed form's launches
    return keep, row, col, val, g


@pytest.mark.parametrize("schedule", [S.SCHEDULE_FUSED, S.SCHEDULE_PIPELINE, S.SCHEDULE_BUFFER])
@pytest.mark.parametrize("K,xdt", [(4, "fp32"), (8, "fp32"), (12, "fp32"), (32, "fp32"), (8, "bf16"), (16, "bf16"),
                                   (24, "bf16"), (64, "bf16"), (72, "bf16"), (136, "bf16"), (256, "bf16"),
                                   (264, "bf16"), (776, "bf16")])
def test_streamed_chunks(graph, K, xdt, schedule):
    n, row, col, val, g = graph
    X = torch.from_numpy(dense_x(n, K, seed=K)).to(DEV).to({"fp32": torch.float32, "bf16": torch.bfloat16}[xdt])
    wide = torch.full((n, K + 4), 7.0, device=DEV)
    g.spmm(X, wide[:, :K], schedule=schedule)
    ref = fp64_reference(n, row, col, val, X.float().cpu().numpy())
    assert rel(wide[:, :K].cpu().numpy(), ref) <= TOL_F32
    assert torch.all(wide[:, K:] == 7.0)
