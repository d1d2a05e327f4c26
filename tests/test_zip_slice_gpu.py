"""A PE's row view whose entries name rows of its own slice only runs on that
slice: nothing before or after the rows that entries name is copied or read."""
import ctypes

import numpy as np
import pytest
import torch

import cola_b200 as cb
from gpu_util import TOL_F32, dense_x, ptr, rel
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("p", [0, 1, 3])
@pytest.mark.parametrize("K", [33, 64, 130])
@pytest.mark.parametrize("per_row", [3, 40])
def test_local_chunks_on_a_slice(p, K, per_row):
    P, n = 4, 4000
    rng = np.random.Generator(np.random.Philox(p))
    npp = n // P
    m = npp * per_row
    lo, hi = p * npp + 100, p * npp + 900  # the columns named: part of the slice
    row = rng.integers(p * npp, (p + 1) * npp, m).astype(np.int32)
    col = rng.integers(lo, hi, m).astype(np.int32)
    val = rng.standard_normal(m).astype(np.float32)
    col[0], col[1] = lo, hi - 1
    g = S.Graph(cb.PartitionSet.from_coo(n, row, col, val, P))
    assert g.nodes_per_part == npp
    z = g.zip_view(p)
    assert z.remote_chunks == 0
    args = [z.csr_rowPtr, z.csr_colIdx, z.csr_rowIdx_zip, z.csr_val, z.csc_colPtr, z.csc_rowIdx, z.csc_colIdx_zip,
            z.csc_val]
    args = [a if a is None or isinstance(a, ctypes.c_void_p) else ctypes.c_void_p(a) for a in args]
    h, L = ctypes.c_void_p(), cb.lib()
    cb._lib.check(L.cola_zip_rows_create(*args, 0, 0, z.local_chunks, 0, npp, p, None, ctypes.byref(h)))
    x = dense_x(npp, K, seed=K)
    xd = torch.from_numpy(x).to(DEV)  # this slice alone
    y = torch.zeros((npp, K), device=DEV)
    size = [ctypes.c_int64(), ctypes.c_int64()]
    cb._lib.check(L.cola_zip_rows_get_info(h, None, None, None, ctypes.byref(size[0])))
    cb._lib.check(L.cola_zip_rows_spmm(h, ptr(y), ptr(xd), K, None))
    cb._lib.check(L.cola_zip_rows_get_info(h, None, None, None, ctypes.byref(size[1])))
    torch.cuda.synchronize()
    L.cola_zip_rows_free(h)
    want = np.zeros((npp, K))
    np.add.at(want, row - p * npp, val[:, None].astype(np.float64) * x[col - p * npp])
    assert rel(y.cpu().numpy(), want) <= TOL_F32
    # no hubs; padded from 16 entries a row of X on: the named rows alone
    padded = (hi - lo) * ((K + 3) // 4) * 16 if K % 4 and m >= 16 * (hi - lo) else 0
    assert size[1].value - size[0].value == padded
