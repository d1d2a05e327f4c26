"""Row-block tasks packed on the device (prep_gpu.cu): the greedy chain is
followed in blocks of 2,048 rows and superblocks of 16 blocks, so the sizes
around their ends, tasks longer than a block, and graphs without and with only
hub rows are compared with the host's row-by-row packing: the same counts, and
the same bits from a width whose float order follows the tasks."""
import numpy as np
import pytest
import torch

import cola_b200 as cb
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BLOCK, SUPER = 2048, 2048 * 16


@pytest.mark.parametrize("n", [1, 2, BLOCK - 1, BLOCK, BLOCK + 1, SUPER - 1, SUPER, SUPER + 1, 3 * SUPER + 77])
@pytest.mark.parametrize("thr,te", [(0, 0), (6, 1), (4, 9), (10 ** 6, 3 * BLOCK), (10 ** 6, 10 ** 7), (1, 40)])
def test_device_tasks_equal_host_tasks(n, thr, te):
    rng = np.random.Generator(np.random.Philox(n * 31 + te + thr))
    # row lengths 0..8, runs of empty rows, a few long rows
    lens = rng.integers(0, 9, n) * (rng.random(n) < 0.6)
    lens[rng.integers(0, n, max(1, n // 500))] = 200
    row = np.repeat(np.arange(n), lens).astype(np.int32)
    col = rng.integers(0, n, len(row)).astype(np.int32)
    val = rng.standard_normal(len(row)).astype(np.float32)
    kw = dict(hub_threshold=thr, hub_segment=32, task_entries=te)
    gd = S.Graph.from_coo_device(n, torch.from_numpy(row).to(DEV), torch.from_numpy(col).to(DEV),
                                 torch.from_numpy(val).to(DEV), nparts=2, **kw)
    gh = S.Graph(cb.PartitionSet.from_coo(n, row, col, val, 2), **kw)
    for k in ("nnz", "hub_rows", "hub_segments", "row_tasks"):
        assert getattr(gd.info, k) == getattr(gh.info, k), k
    X = torch.from_numpy(rng.standard_normal((n, 8)).astype(np.float32)).to(DEV)
    assert torch.equal(gd.spmm(X), gh.spmm(X, schedule=S.SCHEDULE_ROWS))
