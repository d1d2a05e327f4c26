"""k_tile: a tile as wide as K is one pass, the library's own launch (the autotuner's
widest candidate, so that tuning never loses to not tuning); narrower ones are
swept.  Every choice gives the same bits."""
import pytest
import torch

from gpu_util import dense_x, graph_case
from cola_b200 import spmm as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def kernels(g, X, Y, **opts):
    """Names of the kernels one call launches."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        g.spmm(X, Y, **opts)
        torch.cuda.synchronize()
    return " ".join(e.name for e in p.events())


@pytest.mark.parametrize("K,xdt,swept,whole", [(512, torch.float32, (128, 256), (512,)),
                                               (260, torch.float32, (128, 256), (512,)),
                                               (640, torch.float32, (256, 512), ()),
                                               (1024, torch.bfloat16, (256, 512), (1024,)),
                                               (256, torch.bfloat16, (64, 128), (256, 512))])
def test_tile_as_wide_as_k_is_one_pass(K, xdt, swept, whole):
    n, row, col, val, ps = graph_case(11, 16, seed=1, nparts=2)
    g = S.Graph(ps, hub_threshold=64, hub_segment=32)
    X = torch.from_numpy(dense_x(n, K, seed=K)).to(DEV).to(xdt)
    Y = torch.empty((n, K), device=DEV)
    want = g.spmm(X)
    names = kernels(g, X, Y)
    assert "rowblock_spmm" in names and "rowblock_tiled" not in names
    for kt in swept + whole:
        names = kernels(g, X, Y, k_tile=kt)
        assert "rowblock" in names
        assert ("rowblock_tiled" in names) == (kt in swept), kt
        assert torch.equal(g.spmm(X, k_tile=kt), want)
