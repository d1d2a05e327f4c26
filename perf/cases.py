"""Workloads of the partitioned SpMM, each one pass through the package's public entry points.

Graphs are R-MAT (a/b/c/d = 0.57/0.19/0.19/0.05, symmetrised, deduplicated) or uniform random, generated on the
GPU from the seed; values are D^-1/2 A D^-1/2 ("sym") or 1/deg(row) ("row"), features N(0, 1).

Forms ("form" of a case):
  spmm      Graph.spmm on a graph built on the device (the default row-major schedule)
  launcher  ppl0_batch_SpMM once per virtual partition, the kernel-level drop-in on the split blocks
  staged    Graph.spmm with the fused, buffer or pipelined schedule on an uploaded graph
  batch     a captured Batch of graphs of uneven size and width, replayed
  build     a new graph: Graph.from_coo_device on an unsorted edge list, then its first SpMM
  serve     concurrent requests with host features to a Server of resident graphs
"""
import math

import torch

import cola_b200 as cb
from cola_b200 import spmm as S
from cola_b200.batch import Batch
from cola_b200.serving import Server

DEV = "cuda"
DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}
SCHEDULES = {"fused": S.SCHEDULE_FUSED, "buffer": S.SCHEDULE_BUFFER, "pipeline": S.SCHEDULE_PIPELINE}
RMAT = (0.57, 0.19, 0.19)


def listed():
    return [
        # a small graph, one call at a time: launch latency (16 K nodes with self-loops, K = 32)
        dict(name="small-fp32-k32", form="spmm", graph="rmat", n=16384, deg=16.0, loops=True, values="row", parts=4,
             k=32, x="fp32", y="fp32", accumulate=False),
        # the ordinary full-precision product: 1 M nodes, ~31 M entries, K = 128, 8 partitions
        dict(name="fp32-k128", form="spmm", graph="rmat", n=1 << 20, deg=32.0, loops=False, values="sym", parts=8,
             k=128, x="fp32", y="fp32", accumulate=False),
        # the largest: 2 M nodes, ~94 M entries, K = 256, features and output stored BF16
        dict(name="bf16-k256", form="spmm", graph="rmat", n=1 << 21, deg=48.0, loops=False, values="sym", parts=8,
             k=256, x="bf16", y="bf16", accumulate=False),
        # the widest features served
        dict(name="wide-fp32-k512", form="spmm", graph="rmat", n=1 << 18, deg=24.0, loops=False, values="sym",
             parts=8, k=512, x="fp32", y="fp32", accumulate=False),
        # the narrowest features served: BF16 in, FP32 out (class scores, for example)
        dict(name="narrow-bf16-k16", form="spmm", graph="rmat", n=1 << 19, deg=24.0, loops=False, values="sym",
             parts=8, k=16, x="bf16", y="fp32", accumulate=False),
        # Y = B + A X (a residual or bias) on a graph without hubs, sizes that are no power of two
        dict(name="residual-fp32-k100", form="spmm", graph="uniform", n=100003, deg=20.0, loops=False, values="row",
             parts=3, k=100, x="fp32", y="fp32", accumulate=True),
        # a feature width that no vector load divides
        dict(name="odd-fp32-k33", form="spmm", graph="rmat", n=150001, deg=16.0, loops=True, values="sym", parts=4,
             k=33, x="fp32", y="fp32", accumulate=False),
        # many graphs of uneven size in one captured launch
        dict(name="batch-48", form="batch", graphs=48, n_lo=1000, n_hi=200000, deg_lo=4.0, deg_hi=64.0, parts=4,
             x="fp32", y="fp32"),
        # a caller of the kernel-level launcher: zeroed output, one call per partition
        dict(name="launcher-fp32-k128", form="launcher", graph="rmat", n=1 << 18, deg=32.0, loops=False,
             values="sym", parts=8, k=128),
        # the multi-stage work-group schedule
        dict(name="pipeline-bf16-k64", form="staged", schedule="pipeline", graph="rmat", n=1 << 17, deg=32.0,
             loops=False, values="sym", parts=8, group=2, k=64, x="bf16", y="bf16"),
        # a graph that arrives as an edge list and is multiplied once
        dict(name="new-graph", form="build", graph="rmat", n=1 << 20, deg=16.0, loops=False, values="sym", parts=8,
             k=32, x="fp32", y="fp32"),
        # 16 requests at once to 8 resident graphs, widths 16 to 512, half BF16 and half FP32
        dict(name="serve-16", form="serve", graphs=8, scale_lo=12, scale_hi=15, deg_lo=8.0, deg_hi=48.0,
             requests=16),
    ]


# -------------------------------------------------------------------------------------------------------------------
# one more case of the same ranges
# -------------------------------------------------------------------------------------------------------------------
WIDTHS = (16, 32, 64, 100, 128, 256, 512)
SPMM_BYTES = 2.0e10    # gathered bytes of a drawn product: the largest listed one gathers 4.8e10
STAGED_BYTES = 4.0e9   # ... of a drawn product through the chunk schedules, which scatter with atomics


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng):
    return rng.choice(WIDTHS) if rng.random() < 0.6 else _log(rng, 1, 512)


def _fit(c, most):
    """Halve the graph until a pass costs no more than `most` gathered bytes."""
    size = 4 if c.get("x", "fp32") == "fp32" else 2
    if c["k"] * size % 16:
        most /= 4  # no vector loads
    while c["n"] > 1000 and c["n"] * c["deg"] * max(c["k"], 8) * size > most:
        c["n"] = max(1000, c["n"] // 2)
    return c


def draw(rng):
    form = rng.choice(("spmm", "spmm", "spmm", "spmm", "spmm", "batch", "launcher", "staged", "build", "serve"))
    if form == "batch":
        lo = _log(rng, 500, 20000)
        dt = rng.choice(("fp32", "fp32", "bf16"))
        return dict(form=form, graphs=rng.randint(8, 48), n_lo=lo, n_hi=_log(rng, 2 * lo, 200000), deg_lo=4.0,
                    deg_hi=round(rng.uniform(8, 64), 1), parts=rng.choice((1, 2, 4)), x=dt, y=dt)
    if form == "serve":
        lo = rng.randint(10, 14)
        return dict(form=form, graphs=rng.randint(2, 8), scale_lo=lo, scale_hi=rng.randint(lo, 15), deg_lo=8.0,
                    deg_hi=round(rng.uniform(10, 48), 1), requests=rng.randint(1, 16))
    c = dict(form=form, graph=rng.choice(("rmat", "rmat", "rmat", "uniform")), n=_log(rng, 1000, 1 << 21),
             deg=round(rng.uniform(4, 48), 1), loops=rng.random() < 0.5, values=rng.choice(("sym", "row")),
             parts=rng.choice((1, 2, 3, 4, 8)), k=_width(rng))
    if rng.random() < 0.5:
        c["n"] |= 1
    if form == "launcher":
        return _fit(c, STAGED_BYTES)
    c["x"] = rng.choice(("fp32", "bf16"))
    c["y"] = rng.choice((c["x"], "fp32"))
    if form == "spmm":
        c["accumulate"] = c["y"] == "fp32" and rng.random() < 0.25
        return _fit(c, SPMM_BYTES)
    if form == "staged":
        c["schedule"] = rng.choice(("fused", "buffer", "pipeline"))
        c["parts"] = rng.choice((2, 4, 8))
        c["group"] = rng.choice((1, c["parts"] // 2)) if c["schedule"] == "pipeline" else c["parts"]
        return _fit(c, STAGED_BYTES)
    c["k"] = min(c["k"], 128)
    return _fit(c, STAGED_BYTES)


# -------------------------------------------------------------------------------------------------------------------
# inputs
# -------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _edges(gen, graph, n, deg, loops):
    """Distinct symmetric edges as sorted keys row * n + col, and the degree of every row."""
    m = max(1, int(math.ceil(deg * n / 2.0)))
    if graph == "uniform":
        r = torch.randint(0, n, (m,), generator=gen, device=DEV)
        c = torch.randint(0, n, (m,), generator=gen, device=DEV)
    else:
        a, b, cc = RMAT
        r = torch.zeros(m, dtype=torch.int64, device=DEV)
        c = torch.zeros(m, dtype=torch.int64, device=DEV)
        for _ in range(max(1, (n - 1).bit_length())):
            u = torch.rand(m, generator=gen, device=DEV)
            down = u >= a + b
            right = ((u >= a) & ~down) | (u >= a + b + cc)
            r = r * 2 + down
            c = c * 2 + right
        keep = (r < n) & (c < n)  # the subgraph on the first n nodes
        r, c = r[keep], c[keep]
    keep = r != c
    r, c = r[keep], c[keep]
    keys = [r * n + c, c * n + r]
    if loops:
        keys.append(torch.arange(n, device=DEV) * (n + 1))
    keys = torch.unique(torch.cat(keys))
    return keys, torch.bincount(torch.div(keys, n, rounding_mode="floor"), minlength=n)


def _coo(gen, graph, n, deg, loops, values):
    """(row int32, col int32, val float32), sorted by (row, col)."""
    keys, d = _edges(gen, graph, n, deg, loops)
    row = torch.div(keys, n, rounding_mode="floor")
    col = keys - row * n
    d = d.clamp(min=1).double()
    if values == "sym":
        inv = d.rsqrt()
        val = (inv[row] * inv[col]).float()
    else:
        val = (1.0 / d)[row].float()
    return row.int(), col.int(), val


def _case_coo(case, gen):
    return _coo(gen, case["graph"], case["n"], case["deg"], case["loops"], case["values"])


def _features(gen, n, k, dtype):
    return torch.randn((n, k), generator=gen, device=DEV).to(DTYPES[dtype])


def _batch_plan(case, seed):
    """(nodes, degree, width) of every graph of a batch."""
    u = torch.rand((case["graphs"], 3), generator=torch.Generator().manual_seed(int(seed))).tolist()
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    return [(int(round(math.exp(lo + a * (hi - lo)))), case["deg_lo"] + b * (case["deg_hi"] - case["deg_lo"]),
             (32, 64, 128)[int(c * 3)]) for a, b, c in u]


def _serve_plan(case, seed):
    """(nodes, degree) of every resident graph and (graph, width, dtype) of every request."""
    cpu = torch.Generator().manual_seed(int(seed))
    u = torch.rand((case["graphs"], 2), generator=cpu).tolist()
    span = case["scale_hi"] - case["scale_lo"] + 1
    graphs = [(1 << (case["scale_lo"] + int(a * span)), case["deg_lo"] + b * (case["deg_hi"] - case["deg_lo"]))
              for a, b in u]
    v = torch.rand((case["requests"], 3), generator=cpu).tolist()
    reqs = [(int(a * len(graphs)), (16, 64, 256, 512)[int(b * 4)], "fp32" if c < 0.5 else "bf16") for a, b, c in v]
    return graphs, reqs


def _shuffled(gen, row, col, val):
    p = torch.randperm(row.numel(), generator=gen, device=DEV)
    return row[p].contiguous(), col[p].contiguous(), val[p].contiguous()


# A fixed seed for the sizes of batches and request mixes: another seed gives other graphs and features of the same
# sizes.
_PLAN_SEED = 7


def prepare(case, seed):
    gen = _gen(seed)
    form = case["form"]
    st = {"case": case, "form": form}
    if form == "batch":
        graphs, xs, ys = [], [], []
        for n, deg, k in _batch_plan(case, _PLAN_SEED):
            graphs.append(S.Graph.from_coo_device(n, *_coo(gen, "rmat", n, deg, False, "row"), nparts=case["parts"]))
            xs.append(_features(gen, n, k, case["x"]))
            ys.append(torch.empty((n, k), dtype=DTYPES[case["y"]], device=DEV))
        batch = Batch.from_graphs(graphs)
        batch.bind(xs, ys)
        batch.capture()
        st.update(batch=batch, ys=ys)
        return st
    if form == "serve":
        plan, reqs = _serve_plan(case, _PLAN_SEED)
        server = Server(memory_budget=8 << 30)
        for n, deg in plan:
            server.register_graph(S.Graph.from_coo_device(n, *_coo(gen, "rmat", n, deg, False, "sym"), nparts=4))
        st["server"] = server
        st["requests"] = []
        for g, k, dt in reqs:
            x = _features(gen, plan[g][0], k, dt).cpu().pin_memory()
            st["requests"].append((g, x, torch.empty_like(x).pin_memory()))
        return st
    n, k = case["n"], case["k"]
    row, col, val = _case_coo(case, gen)
    if form == "build":
        st.update(n=n, coo=_shuffled(gen, row, col, val), x=_features(gen, n, k, case["x"]))
        return st
    if form == "spmm":
        st["graph"] = S.Graph.from_coo_device(n, row, col, val, nparts=case["parts"])
        st["x"] = _features(gen, n, k, case["x"])
        st["y"] = torch.empty((n, k), dtype=DTYPES[case["y"]], device=DEV)
        if case["accumulate"]:
            st["bias"] = _features(gen, n, k, "fp32")
        return st
    pset = cb.PartitionSet.from_coo_device(n, row, col, val, nparts=case["parts"])
    if form == "staged":
        st["graph"] = S.Graph(pset, group_size=case["group"])
        st["x"] = _features(gen, n, k, case["x"])
        st["y"] = torch.empty((n, k), dtype=DTYPES[case["y"]], device=DEV)
        return st
    g = S.Graph(pset)
    npp = g.nodes_per_part
    x = torch.zeros((case["parts"] * npp, k), device=DEV)
    x[:n] = _features(gen, n, k, "fp32")
    st.update(graph=g, zips=[g.zip_view(p) for p in range(case["parts"])], x=x,
              y=torch.empty((case["parts"] * npp, k), device=DEV))
    return st


# -------------------------------------------------------------------------------------------------------------------
# one pass
# -------------------------------------------------------------------------------------------------------------------
def run(state):
    form, case = state["form"], state["case"]
    if form == "spmm":
        if case["accumulate"]:
            state["y"].copy_(state["bias"])
        return state["graph"].spmm(state["x"], state["y"], accumulate=case["accumulate"])
    if form == "batch":
        state["batch"].replay()
        return state["ys"]
    if form == "launcher":
        x, y, g = state["x"], state["y"], state["graph"]
        npp, k = g.nodes_per_part, case["k"]
        y.zero_()
        for p, z in enumerate(state["zips"]):
            at = p * npp * k * 4
            S.ppl0_batch_SpMM(y.data_ptr() + at, x.data_ptr() + at, z.csr_rowPtr, z.csr_colIdx, z.csr_rowIdx_zip,
                              z.csr_val, z.csc_colPtr, z.csc_rowIdx, z.csc_colIdx_zip, z.csc_val, 0, 0,
                              z.local_chunks, z.remote_chunks, k, npp, p)
        return y
    if form == "staged":
        return state["graph"].spmm(state["x"], state["y"], schedule=SCHEDULES[case["schedule"]])
    if form == "build":
        graph = S.Graph.from_coo_device(state["n"], *state["coo"], nparts=case["parts"])
        return graph.spmm(state["x"], out_dtype=DTYPES[case["y"]])
    reqs = [state["server"].submit(g, x, out_dtype=x.dtype, Y=y) for g, x, y in state["requests"]]
    return [r.wait() for r in reqs]


# -------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and its result in 64 bits
# -------------------------------------------------------------------------------------------------------------------
def _products(case):
    """(entries, nodes, width, bytes per feature in, bytes per feature out) of every product of a pass; the entries
    as drawn, before duplicates and self-loops are dropped."""
    size = {"fp32": 4, "bf16": 2}
    if case["form"] == "batch":
        return [(deg * n, n, k, size[case["x"]], size[case["y"]]) for n, deg, k in _batch_plan(case, _PLAN_SEED)]
    if case["form"] == "serve":
        plan, reqs = _serve_plan(case, _PLAN_SEED)
        return [(plan[g][0] * plan[g][1], plan[g][0], k, size[dt], size[dt]) for g, k, dt in reqs]
    n = case["n"]
    return [(n * (case["deg"] + (1 if case["loops"] else 0)), n, case["k"], size[case.get("x", "fp32")],
             size[case.get("y", "fp32")])]


def work(case):
    total, flops = 0.0, 0.0
    for nnz, n, k, sx, sy in _products(case):
        # column ids and values, row pointers, X once, Y once
        total += nnz * 8 + (n + 1) * 4 + n * k * (sx + sy)
        flops += 2.0 * nnz * k
        if case.get("accumulate"):
            total += n * k * 4  # the residual
        if case["form"] == "build":
            total += nnz * 12   # the edge list
    return {"bytes": total, "flops": flops}


def _exact(n, row, col, val, x):
    """A X in 64 bits, from the entries sorted by row."""
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    a = torch.sparse_csr_tensor(ptr, col.long(), val.double(), size=(n, n))
    return a @ x.double()


def exact(case, seed):
    gen = _gen(seed)
    form = case["form"]
    if form == "batch":
        out = []
        for n, deg, k in _batch_plan(case, _PLAN_SEED):
            coo = _coo(gen, "rmat", n, deg, False, "row")
            out.append(_exact(n, *coo, _features(gen, n, k, case["x"])))
        return out
    if form == "serve":
        plan, reqs = _serve_plan(case, _PLAN_SEED)
        coos = [_coo(gen, "rmat", n, deg, False, "sym") for n, deg in plan]
        return [_exact(plan[g][0], *coos[g], _features(gen, plan[g][0], k, dt)).cpu() for g, k, dt in reqs]
    n, k = case["n"], case["k"]
    row, col, val = _case_coo(case, gen)
    if form == "build":
        _shuffled(gen, row, col, val)
    y = _exact(n, row, col, val, _features(gen, n, k, case.get("x", "fp32")))
    if form == "spmm" and case["accumulate"]:
        y += _features(gen, n, k, "fp32").double()
    if form == "launcher":
        rows = case["parts"] * (-(-n // case["parts"]))
        y = torch.cat([y, torch.zeros((rows - n, k), dtype=torch.float64, device=DEV)])
    return y
