"""Freeing a graph, or building one, while a stream is being captured leaves the
capture alone, waits for the graph's running products and gives its memory back."""
import threading

import pytest
import torch

import cola_b200 as cb
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def edges(n, m, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    r = [torch.randint(0, n, (m,), generator=g, device=DEV, dtype=torch.int32) for _ in range(2)]
    return r[0], r[1], torch.rand(m, generator=g, device=DEV)


@pytest.mark.parametrize("mode,thread", [("thread_local", True), ("relaxed", True), ("global", True),
                                         ("thread_local", False), ("global", False)])
def test_free_during_a_capture(mode, thread):
    n, m = 50000, 1 << 24
    coo = edges(n, m, 1)
    g = S.Graph.from_coo_device(n, *coo)
    x = torch.randn((n, 32), device=DEV)
    g.spmm(x)
    g.close()
    assert cb.lib().cola_trim_memory() == 0
    g = S.Graph.from_coo_device(n, *coo)
    a = torch.arange(1000, dtype=torch.float32, device=DEV)
    b = torch.zeros_like(a)
    torch.cuda.synchronize()
    assert cb.lib().cola_trim_memory() == 0
    before = torch.cuda.mem_get_info()[0]
    cg = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cg, capture_error_mode=mode):
        torch.mul(a, 2, out=b)
        if thread:
            t = threading.Thread(target=g.close)
            t.start()
            t.join()
        else:
            g.close()
        b.add_(1)
    cg.replay()
    torch.cuda.synchronize()
    assert torch.equal(b, 2 * a + 1)
    assert cb.lib().cola_trim_memory() == 0
    # the graph's columns and values at least; chunks at its ends may be shared with
    # graphs that are alive
    assert torch.cuda.mem_get_info()[0] - before >= m * 8 - (64 << 20) > 0


def test_free_waits_for_running_products():
    n = 20000
    g = S.Graph.from_coo_device(n, *edges(n, 200000, 2))
    x = torch.randn((n, 16), device=DEV)
    want = g.spmm(x)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        torch.cuda._sleep(20_000_000)  # about 10 ms
        y = g.spmm(x, stream=st)
    assert not st.query()
    g.close()
    assert st.query()
    assert torch.equal(y, want)
