"""device_bytes of a graph, a batch and a row view of zip arrays count every
workspace, the padded copy of X among them."""
import ctypes

import numpy as np
import pytest
import torch

import cola_b200 as cb
from gpu_util import dense_x, ptr
from cola_b200 import spmm as S
from cola_b200.batch import Batch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_padded_copies_are_counted():
    rng = np.random.Generator(np.random.Philox(3))
    n, m = 2000, 80000  # 40 entries a row: padded copies are made, no hubs
    row, col = (rng.integers(0, n, m).astype(np.int32) for _ in range(2))
    ps = cb.PartitionSet.from_coo(n, row, col, rng.standard_normal(m).astype(np.float32), 1)
    g = S.Graph(ps)
    assert g.info.hub_rows == 0 and col.min() == 0 and col.max() == n - 1
    padded = n * 9 * 16  # rows of 33 floats
    b = Batch.from_graphs([g])
    before = g.get_info().device_bytes, b.info.device_bytes
    x = torch.from_numpy(dense_x(n, 33, seed=1)).to(DEV)
    g.spmm(x)
    assert g.get_info().device_bytes == before[0] + padded
    assert b.info.device_bytes == before[1] + padded
    z = g.zip_view(0)
    h = ctypes.c_void_p()
    L = cb.lib()
    args = [z.csr_rowPtr, z.csr_colIdx, z.csr_rowIdx_zip, z.csr_val, z.csc_colPtr, z.csc_rowIdx, z.csc_colIdx_zip,
            z.csc_val]
    args = [a if a is None or isinstance(a, ctypes.c_void_p) else ctypes.c_void_p(a) for a in args]
    cb._lib.check(L.cola_zip_rows_create(*args, 0, 0, z.local_chunks, z.remote_chunks, g.nodes_per_part, 0, None,
                                         ctypes.byref(h)))
    size = [ctypes.c_int64(), ctypes.c_int64()]
    y = torch.zeros((n, 33), device=DEV)
    cb._lib.check(L.cola_zip_rows_get_info(h, None, None, None, ctypes.byref(size[0])))
    cb._lib.check(L.cola_zip_rows_spmm(h, ptr(y), ptr(x), 33, None))
    cb._lib.check(L.cola_zip_rows_get_info(h, None, None, None, ctypes.byref(size[1])))
    torch.cuda.synchronize()
    L.cola_zip_rows_free(h)
    assert size[1].value == size[0].value + padded
    b.close()
