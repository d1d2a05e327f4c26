"""The device sort behind the partition and graph builds: sizes around the
4,096-entry tile and the 512 entries of a warp, key widths of 0 to 6 digits, all
entries in one row or one column, many duplicates, against the host build."""
import numpy as np
import pytest
import torch

import cola_b200 as cb
from gpu_util import TOL_F32, dense_x, fp64_reference, rel
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nnz", [1, 31, 511, 512, 513, 4095, 4096, 4097, 20000])
@pytest.mark.parametrize("n,kind", [(1, "any"), (2, "any"), (200, "any"), (70000, "any"), (5000000, "any"),
                                    (300, "row"), (300, "col"), (9, "dups")])
def test_partitions_equal_host(n, kind, nnz):
    rng = np.random.Generator(np.random.Philox(nnz + n))
    row = rng.integers(0, n, nnz).astype(np.int32)
    col = rng.integers(0, n, nnz).astype(np.int32)
    if kind == "row":
        row[:] = 5
    if kind == "col":
        col[:] = 299
    val = rng.standard_normal(nnz).astype(np.float32)
    P = 3 if n > 2 else 1
    t = [torch.from_numpy(a).to(DEV) for a in (row, col, val)]
    for v_dev, v_host in ((t[2], val), (None, None)):
        d = cb.PartitionSet.from_coo_device(n, t[0], t[1], v_dev, P)
        h = cb.PartitionSet.from_coo(n, row, col, v_host, P)
        for r in range(P):
            a, b = d.part(r), h.part(r)
            for k in a:
                assert np.array_equal(np.asarray(a[k]), np.asarray(b[k])), (k, r)
    if n <= 70000:
        g = S.Graph.from_coo_device(n, *t, nparts=P)
        X = dense_x(n, 12, seed=n)
        ref = fp64_reference(n, row, col, val, X)
        assert rel(g.spmm(torch.from_numpy(X).to(DEV)).cpu().numpy(), ref) <= TOL_F32
