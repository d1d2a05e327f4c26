"""The library's memory pool: freed graphs' memory is kept within its bound and
given back by cola_trim_memory; graphs built by several threads on streams of
their own, while others are freed, are right."""
import threading

import numpy as np
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


def test_freed_memory_is_bounded_and_given_back():
    n, m = 100000, 1 << 23
    coo = edges(n, m, 1)
    torch.cuda.synchronize()
    assert cb.lib().cola_trim_memory() == 0
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        g = S.Graph.from_coo_device(n, *coo)
        g.close()
    torch.cuda.synchronize()
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert kept <= (1 << 30) + (64 << 20)
    assert cb.lib().cola_trim_memory() == 0
    assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20


def test_builds_and_frees_from_several_threads():
    n, m, K = 20000, 300000, 40
    coos = [edges(n, m, s) for s in range(4)]
    x = torch.randn((n, K), device=DEV)
    want = [S.Graph.from_coo_device(n, *c).spmm(x) for c in coos]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            for rep in range(6):
                c = coos[(i + rep) % 4]
                g = S.Graph.from_coo_device(n, *c, stream=st)
                y = g.spmm(x, stream=st)
                g.close()  # with the product still running
                st.synchronize()
                if not torch.equal(y, want[(i + rep) % 4]):
                    bad.append((i, rep))
    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
