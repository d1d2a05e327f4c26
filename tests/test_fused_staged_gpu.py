"""The streamed form of the fused kernel on remote rows staged in device memory: a
buffer batch, and a later pipeline stage, with chunks enough in one launch (4
blocks of 8 warps on each of 148 multiprocessors, half a span of 8 chunks a
warp), and launches one batch row short of that, against FP64."""
import pytest
import torch

import cola_b200 as cb
from gpu_util import TOL_F32, dense_x, fp64_reference, rel
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
STREAMS = 148 * 4 * 8 * 4  # chunks of a launch from which it is streamed


@pytest.fixture(scope="module")
def graph():
    n, row, col, val = cb.rmat(17, 10, seed=2)
    keep = n - 5
    m = (row < keep) & (col < keep)
    row, col, val = row[m], col[m], val[m]
    g = S.Graph(cb.PartitionSet.from_coo(keep, row, col, val, 2), group_size=1)
    remote = [g.zip_view(p).remote_chunks for p in range(2)]
    assert max(remote) > STREAMS + 100
    return keep, row, col, val, g, remote


@pytest.mark.parametrize("rows", [1 << 16, STREAMS, STREAMS - 1])
@pytest.mark.parametrize("K,xdt", [(4, "fp32"), (32, "fp32"), (8, "bf16"), (24, "bf16"), (64, "bf16"), (136, "bf16")])
def test_buffer_batches(graph, K, xdt, rows):
    n, row, col, val, g, remote = graph
    # at least one batch has `rows` chunks, or all of its partition's
    assert max(min(r, rows) for r in remote) >= STREAMS - 1
    check(graph, K, xdt, S.SCHEDULE_BUFFER, rows)


@pytest.mark.parametrize("K,xdt", [(8, "fp32"), (32, "fp32"), (16, "bf16"), (64, "bf16"), (264, "bf16")])
def test_pipeline_stage(graph, K, xdt):
    # two partitions, groups of one: the only later stage launches every remote chunk
    assert sum(graph[5]) >= STREAMS
    check(graph, K, xdt, S.SCHEDULE_PIPELINE, 0)


def check(graph, K, xdt, schedule, rows):
    n, row, col, val, g, remote = graph
    X = torch.from_numpy(dense_x(n, K, seed=K)).to(DEV).to({"fp32": torch.float32, "bf16": torch.bfloat16}[xdt])
    wide = torch.full((n, K + 4), 7.0, device=DEV)
    g.spmm(X, wide[:, :K], schedule=schedule, gather_batch_rows=rows)
    ref = fp64_reference(n, row, col, val, X.float().cpu().numpy())
    assert rel(wide[:, :K].cpu().numpy(), ref) <= TOL_F32
    assert torch.all(wide[:, K:] == 7.0)
