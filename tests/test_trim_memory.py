"""cola_b200.trim_memory: callable without a GPU; on one, what a freed graph left in
the pool is free memory of the device again."""
import pytest

import cola_b200 as cb


def test_without_graphs():
    assert cb.trim_memory() is None


@pytest.mark.gpu
def test_gives_back_what_a_freed_graph_left():
    import torch
    from cola_b200 import spmm as S
    n, m = 100000, 1 << 24
    gen = torch.Generator(device="cuda:0")
    gen.manual_seed(1)
    r, c = (torch.randint(0, n, (m,), generator=gen, device="cuda:0", dtype=torch.int32) for _ in range(2))
    g = S.Graph.from_coo_device(n, r, c)
    held = g.get_info().device_bytes
    g.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    cb.trim_memory()
    # chunks at its ends may be shared with graphs that are alive
    assert torch.cuda.mem_get_info()[0] - before >= held - (64 << 20) > 0
