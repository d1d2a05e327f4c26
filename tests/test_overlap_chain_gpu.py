"""Row-major products chained through each other's outputs with nothing between
them: up to three launches are resident at once, each reads what the one before
it wrote into memory that the one before that read.  Equal to one at a time."""
import numpy as np
import pytest
import torch

import cola_b200 as cb
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def chain(g, x0, sync, accumulate):
    x, y = x0.clone(), torch.zeros_like(x0)
    torch.cuda.synchronize()
    for s in range(20):
        g.spmm(x, y, accumulate=accumulate and s % 3 == 1)
        sync()
        g.spmm(y, x, accumulate=accumulate and s % 2 == 1)
        sync()
    torch.cuda.synchronize()
    return x, y


@pytest.mark.parametrize("scale", [7, 9, 11, 13])
@pytest.mark.parametrize("hubs", [True, False])
@pytest.mark.parametrize("K,dt", [(4, "fp32"), (33, "fp32"), (36, "fp32"), (128, "fp32"), (8, "bf16"), (264, "bf16")])
def test_ping_pong(scale, hubs, K, dt):
    n, row, col, _ = cb.rmat(scale, 10, seed=scale)
    val = (1.0 / np.bincount(row, minlength=n).clip(1)[row]).astype(np.float32)  # rows sum to 1: no growth
    g = S.Graph(cb.PartitionSet.from_coo(n, row, col, val, 2), hub_threshold=8 if hubs else 10 ** 6)
    x0 = torch.randn((n, K), device=DEV).to({"fp32": torch.float32, "bf16": torch.bfloat16}[dt])
    for accumulate in ([False, True] if dt == "fp32" else [False]):
        want = chain(g, x0, torch.cuda.synchronize, accumulate)
        for rep in range(5):
            got = chain(g, x0, lambda: None, accumulate)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
