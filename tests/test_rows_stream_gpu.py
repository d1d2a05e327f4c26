"""The row-major schedule's work items and hub combine at the sizes where they
can go wrong: rows that end on, before and after a 32-entry batch, a round of
every lane geometry, runs of empty rows, graphs without and with only hubs, and
hubs of every number of partials around the powers of the combine's radix (8)
and its shared-by-a-block threshold (32), against FP64; the batched form gives
the same bits."""
import numpy as np
import pytest
import torch

from gpu_util import TOL_F32, dense_x, fp64_reference, rel
from cola_b200 import spmm as S
from cola_b200.batch import Batch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def graph(lens, ncol, seed, **kw):
    rng = np.random.Generator(np.random.Philox(seed))
    n = len(lens)
    row = np.repeat(np.arange(n), lens).astype(np.int32)
    col = np.concatenate([rng.choice(ncol, l, replace=False) if l <= ncol else rng.integers(0, ncol, l)
                          for l in lens] + [np.zeros(0, np.int64)]).astype(np.int32)
    val = rng.standard_normal(len(row)).astype(np.float32)
    g = S.Graph.from_coo_device(n, torch.from_numpy(row).to(DEV), torch.from_numpy(col).to(DEV),
                                torch.from_numpy(val).to(DEV), nparts=2, **kw)
    return n, row, col, val, g


CASES = {
    "edges": ([0, 0, 1, 31, 32, 33, 0, 63, 64, 65, 2, 30, 7, 8, 9, 0] * 20, {}),
    "no entries": ([0] * 70, {}),
    "one row": ([5], {}),
    "hubs": ([1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 71, 255, 256, 257, 511, 512, 513, 520, 600],
             dict(hub_threshold=0, hub_segment=1)),
    "only hubs": ([600] * 8, dict(hub_threshold=4, hub_segment=5)),
    "long task": ([3] * 700 + [0] * 50 + [100] * 3, dict(hub_threshold=10 ** 6, hub_segment=7, task_entries=5000)),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("K,xdt,ydt", [(4, "fp32", "fp32"), (8, "bf16", "bf16"), (12, "fp32", "bf16"),
                                       (16, "bf16", "fp32"), (32, "fp32", "fp32"), (64, "bf16", "bf16"),
                                       (64, "fp32", "fp32"), (128, "bf16", "fp32"), (132, "fp32", "fp32"),
                                       (256, "bf16", "bf16"), (520, "bf16", "fp32"), (1028, "fp32", "fp32")])
def test_items_and_combine(name, K, xdt, ydt):
    lens, kw = CASES[name]
    kw = dict(kw)
    if kw.get("hub_threshold") == 0:  # 0 means the default: every row a hub
        kw["hub_threshold"] = 1
    lens = list(lens) + [0] * (700 - len(lens))  # at least as many columns as the longest row
    n, row, col, val, g = graph(lens, len(lens), 5, **kw)
    dt = {"fp32": torch.float32, "bf16": torch.bfloat16}
    X = torch.from_numpy(dense_x(n, K, seed=K)).to(DEV).to(dt[xdt])
    ref = fp64_reference(n, row, col, val, X.float().cpu().numpy())
    Y = torch.full((n, K), float("nan"), device=DEV).to(dt[ydt])
    g.spmm(X, Y)
    Y32 = torch.full((n, K), float("nan"), device=DEV)
    g.spmm(X, Y32)
    got = Y32.cpu().numpy()
    if ref.any():
        assert rel(got, ref) <= TOL_F32
    else:
        assert not got.any()
    assert torch.equal(Y, Y32.to(dt[ydt]))  # a BF16 output is the FP32 sums, rounded once
    b = Batch.from_graphs([g, g])
    Ys = [torch.full_like(Y, float("nan")) for _ in range(2)]
    b.bind([X, X], Ys)
    b.run()
    assert torch.equal(Ys[0], Y) and torch.equal(Ys[1], Y)
    if ydt == "fp32":
        B = torch.from_numpy(dense_x(n, K, seed=K + 1)).to(DEV)
        Z = B.clone()
        g.spmm(X, Z, accumulate=True)
        assert torch.equal(Z, B + Y)
