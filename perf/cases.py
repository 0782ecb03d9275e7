"""The work that users of this library give it, as timed cases.

A case is a dict of plain values.  `prepare` makes what a program holds before
the call (a loaded graph, a committed batch, a started server, a packed BVSS,
a device array), `run` makes one pass through the public entry points, `work`
counts what a pass cannot do without, and `exact` gives the costs in 64-bit
arithmetic from plain torch.

The graphs are seeded levelised timing DAGs of the shapes that the tests and
the benchmark use: pins in levels, edges to the next `span` levels, a
super-source before the first level and a super-sink after the last, vertex
ids without level order.  They are made on the GPU, since they are made often.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-cpg_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cpg_b200  # noqa: E402

DEV = "cuda"
SCALE = 10000.0  # fixed-point units per delay unit in the suffix tree


def listed():
    return [
        # Signoff of one block: the smallest query, bound by latency and launches.
        dict(name="query_20k", kind="query", pins=20_000, levels=60, span=3, degree="uniform",
             mean=2.5, integer=False, k=1_000),
        # An ordinary block, odd sizes.
        dict(name="query_100k", kind="query", pins=100_003, levels=97, span=3, degree="geometric",
             mean=5.0, integer=False, k=20_011),
        # The headline query: a full design, a million paths.
        dict(name="query_1m", kind="query", pins=1_000_000, levels=200, span=4, degree="geometric",
             mean=20.0, integer=False, k=1_000_000),
        # The dense end of the degree sweep: most of the time is the suffix tree's.
        dict(name="query_1m_dense", kind="query", pins=1_000_000, levels=200, span=4,
             degree="geometric", mean=50.0, integer=False, k=100_000),
        # A second report on a graph whose suffix tree is current: the enumeration alone,
        # with integer delays (many tied costs).
        dict(name="requery_400k_int", kind="requery", pins=400_000, levels=200, span=4,
             degree="geometric", mean=10.0, integer=True, k=200_000),
        # A what-if loop: 1% of the delays change, report, change back, report.
        dict(name="whatif_200k", kind="whatif", pins=200_001, levels=120, span=3,
             degree="geometric", mean=8.0, integer=False, k=10_000),
        # A graph that arrives from the host: upload, build and report in one pass.
        dict(name="load_300k", kind="load", pins=300_000, levels=150, span=4, degree="geometric",
             mean=20.0, integer=False, k=100_000),
        # The batched form: many blocks of uneven size in one captured step.
        dict(name="batch_48", kind="batch", graphs=48, mix=4, rebuild=True),
        # The served form: requests over resident graphs, some with delay updates.
        dict(name="serve_48", kind="serve", graphs=12, mix=5, requests=48),
        # BFS levels over bit slices, and deviation pairs of a source set.
        dict(name="bvss_levels_200k", kind="bvss_levels", levels=100, width=2_000, deg=16,
             window=24),
        dict(name="bvss_pairs_100k", kind="bvss_pairs", levels=100, width=1_000, deg=16, window=24,
             sources=20_000),
        # The K cheapest of a device array of path costs, as an operator of its own.
        dict(name="topk_8m", kind="topk", n=8_000_000, k=200_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "requery", "whatif", "load", "batch", "serve",
                       "bvss_levels", "bvss_pairs", "topk"])
    if kind in ("query", "requery", "whatif", "load"):
        pins = _log(rng, 20_000, {"query": 1_000_000, "requery": 1_000_000}.get(kind, 400_000))
        mean = math.exp(rng.uniform(math.log(2.5), math.log(min(50.0, 2e7 / pins))))
        top = min(10 * pins, 1_000_000 if kind in ("query", "requery") else 100_000)
        return dict(kind=kind, pins=pins, levels=rng.randint(40, 200), span=rng.choice([3, 4]),
                    degree="geometric", mean=round(mean, 2), integer=rng.random() < 0.25,
                    k=_log(rng, 1_000, top))
    if kind == "batch":
        return dict(kind=kind, graphs=rng.randint(4, 40), mix=rng.randrange(1 << 20), rebuild=rng.random() < 0.7)
    if kind == "serve":
        return dict(kind=kind, graphs=rng.randint(4, 12), mix=rng.randrange(1 << 20),
                    requests=rng.randint(8, 48))
    if kind == "bvss_levels":
        deg = rng.randint(4, 16)
        return dict(kind=kind, levels=rng.randint(40, 120), width=_log(rng, 200, 2_000), deg=deg,
                    window=rng.randint(deg, 24))
    if kind == "bvss_pairs":
        deg, width = rng.randint(4, 16), _log(rng, 100, 1_000)
        return dict(kind=kind, levels=100, width=width, deg=deg, window=rng.randint(deg, 24),
                    sources=_log(rng, 100, 20 * width))
    n = _log(rng, 10_000, 8_000_000)
    return dict(kind=kind, n=n, k=_log(rng, 100, min(200_000, n // 2)))


# ------------------------------------------------------------------ graphs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


class _Graph:
    """Fan-out CSR on the GPU, with each vertex's place in level order."""

    def __init__(self, seed, pins, levels, span, degree, mean, integer, cap=256):
        g = _gen(seed)
        side = min(2_000, max(8, pins // (2 * levels)))
        sizes = torch.full((levels,), (pins - 2 * side) // (levels - 2), dtype=torch.int64)
        sizes[1:1 + (pins - 2 * side) % (levels - 2)] += 1
        sizes[0] = sizes[-1] = side
        start = torch.zeros(levels + 1, dtype=torch.int64)
        start[1:] = torch.cumsum(sizes, 0)
        self.bounds = [0] + [int(x) + 1 for x in start] + [pins + 2]  # super-source, levels, super-sink
        start = start.to(DEV)
        level = torch.repeat_interleave(torch.arange(levels, device=DEV), sizes.to(DEV))
        inner = int(start[levels - 1])  # pins below the last level have fan-out
        if degree == "uniform":
            deg = torch.randint(1, int(2 * mean), (inner,), generator=g, device=DEV)
        else:
            u = torch.rand(inner, generator=g, device=DEV, dtype=torch.float64).clamp_(min=1e-300)
            deg = (1 + torch.floor(torch.log(u) / math.log(1 - 1 / mean))).clamp_(max=cap).long()
        src = torch.repeat_interleave(torch.arange(inner, device=DEV), deg)
        lv = level[src]
        hop = torch.minimum((levels - 1) - lv, torch.tensor(span, device=DEV))
        to = lv + 1 + torch.floor(torch.rand(src.numel(), generator=g, device=DEV) * hop).long().clamp_(max=span - 1)
        to = torch.minimum(to, torch.tensor(levels - 1, device=DEV))
        width = start[to + 1] - start[to]
        at = torch.floor(torch.rand(src.numel(), generator=g, device=DEV) * width).long()
        dst = start[to] + torch.minimum(at, width - 1)
        # a pin without fan-in gets an edge from the level before
        lone = torch.nonzero(torch.bincount(dst, minlength=pins)[side:] == 0).flatten() + side
        lv = level[lone] - 1
        width = start[lv + 1] - start[lv]
        at = torch.floor(torch.rand(lone.numel(), generator=g, device=DEV) * width).long()
        first, last = torch.arange(side, device=DEV), torch.arange(pins - side, pins, device=DEV)
        src = torch.cat([src, start[lv] + torch.minimum(at, width - 1), torch.full_like(first, pins), last])
        dst = torch.cat([dst, lone, first, torch.full_like(last, pins + 1)])
        n = pins + 2
        ids = torch.randperm(pins, generator=g, device=DEV)
        ids = torch.cat([ids, torch.tensor([pins, pins + 1], device=DEV)])
        key = torch.unique(ids[src] * n + ids[dst])
        src = key // n
        self.n, self.adj = n, (key % n).int()
        self.adjp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
        self.adjp[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
        self.integer = integer
        self.free = (src == pins) | (self.adj == pins + 1)  # the virtual edges have no delay
        self.w = self.delays(g, key.numel())
        self.w[self.free] = 0.0
        # vertex ids in level order: super-source, pins, super-sink
        self.order = torch.cat([ids[pins:pins + 1], ids[:pins], ids[pins + 1:]])

    def delays(self, g, count):
        if self.integer:
            return torch.randint(1, 101, (count,), generator=g, device=DEV).float()
        return 0.1 + 9.9 * torch.rand(count, generator=g, device=DEV)

    def change(self, seed):
        """1% of the edges with new delays, and the same edges as they are."""
        g = _gen(seed)
        real = torch.nonzero(~self.free).flatten()
        e = real[torch.randperm(real.numel(), generator=g, device=DEV)[:max(1, real.numel() // 100)]]
        return e, self.delays(g, e.numel()), self.w[e]

    def host(self):
        return self.n, self.adjp.int().cpu().numpy(), self.adj.cpu().numpy(), self.w.cpu().numpy()

    def lowest(self, k, w=None):
        """The k lowest path costs in 64 bits.  Suffix-tree edges cost their fixed-point
        delay, every other edge its delay.  A partial path's bound is its cost with the
        suffix tree's rest, so the k lowest bounds of each step are all that is kept."""
        w = self.w if w is None else w
        adjp, adj = self.adjp, self.adj.long()
        fixed = (w * SCALE).to(torch.int32).long()
        dist = torch.full((self.n,), 1 << 40, dtype=torch.int64, device=DEV)
        succ = torch.full((self.n,), -1, dtype=torch.int64, device=DEV)
        dist[self.order[-1]] = 0
        for lo, hi in zip(self.bounds[-3::-1], self.bounds[-2:0:-1]):
            v = self.order[lo:hi]
            row, e = self._edges(v)
            c = dist[adj[e]] + fixed[e]
            d = torch.full((v.numel(),), 1 << 40, dtype=torch.int64, device=DEV).scatter_reduce_(0, row, c, "amin")
            s = torch.full((v.numel(),), -1, dtype=torch.int64, device=DEV)
            s.scatter_reduce_(0, row, torch.where(c == d[row], adj[e], -1), "amax")
            dist[v], succ[v] = d, s
        real = dist.double() / SCALE
        at = self.order[:1]
        f = real[at].clone()
        done, limit = f[:0], math.inf
        while at.numel():
            row, e = self._edges(at)
            head = adj[e]
            tail = at[row]
            c = f[row] + torch.where(head == succ[tail], 0.0, real[head] + w[e].double() - real[tail])
            keep = c <= limit
            at, f = head[keep], c[keep]
            end = adjp[at + 1] == adjp[at]
            done = torch.cat([done, f[end]])
            at, f = at[~end], f[~end]
            every = torch.cat([done, f])
            if every.numel() > k:
                low, which = torch.topk(every, k, largest=False)
                limit = float(low.max())
                inner = which[which >= done.numel()] - done.numel()
                done = done[which[which < done.numel()]]
                at, f = at[inner], f[inner]
        return torch.sort(done)[0][:k].cpu()

    def _edges(self, v):
        """(index into v, edge id) of every edge leaving the vertices v."""
        deg = self.adjp[v + 1] - self.adjp[v]
        row = torch.repeat_interleave(torch.arange(v.numel(), device=DEV), deg)
        first = torch.cumsum(deg, 0) - deg
        return row, self.adjp[v][row] + torch.arange(row.numel(), device=DEV) - first[row]


def _graph(case, seed):
    return _Graph(seed, case["pins"], case["levels"], case["span"], case["degree"], case["mean"],
                  case["integer"])


def _blocks(case, most):
    """Sizes of the blocks of a batched or served case: pins log-uniform from 5,000, mean degree
    2-8.  Part of the case (its mix); edges and delays are the seed's."""
    rng = random.Random(case["mix"])
    got = []
    for _ in range(case["graphs"]):
        got.append(dict(pins=_log(rng, 5_000, most), levels=rng.randint(40, 150), span=3,
                        degree="geometric", mean=rng.uniform(2.0, 8.0), integer=False, cap=64))
    return got


def _batch_ks(case):
    rng = random.Random(case["mix"] + 1)
    return [_log(rng, 100, 100_000) for _ in range(case["graphs"])]


def _requests(case):
    """(graph, k, change) of each request: on every other graph one request changes 1% of the
    delays first (change 1) and the last one changes them back (change 0), so a pass leaves the
    graphs as it found them; None changes nothing."""
    rng = random.Random(case["mix"] + 2)
    got = [[rng.randrange(case["graphs"]), _log(rng, 100, 20_000), None] for _ in range(case["requests"])]
    for g in range(0, case["graphs"], 2):
        mine = [r for r in got if r[0] == g]
        if len(mine) >= 2:
            mine[len(mine) // 3][2] = 1
            mine[-1][2] = 0
    return [tuple(r) for r in got]


def _local(case, seed):
    """Rows whose heads lie in a window of pins of one of the next three levels (dense slices),
    on the host."""
    g = _gen(seed)
    levels, width, deg, span = case["levels"], case["width"], case["deg"], case["window"]
    rows = (levels - 1) * width
    hop = torch.randint(1, 4, (rows,), generator=g, device=DEV)
    base = (torch.arange(rows, device=DEV) // width + hop).clamp_(max=levels - 1) * width
    off = torch.randint(0, width - span + 1, (rows,), generator=g, device=DEV)
    pick = torch.argsort(torch.rand(rows, span, generator=g, device=DEV), dim=1)[:, :deg]
    adj = (base + off)[:, None] + pick
    n = levels * width
    adjp = torch.arange(n + 1, device=DEV).clamp_(max=rows) * deg
    return n, adjp.int().cpu().numpy(), adj.int().flatten().cpu().numpy(), rows * deg, g


# ------------------------------------------------------------------ the cases
def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind)
    if kind in ("query", "requery", "whatif", "load"):
        gr = _graph(case, seed)
        s["k"] = case["k"]
        h = s["handle"] = cpg_b200.CpGen()
        if kind == "load":
            n, *arrays = gr.host()
            s["csr"] = [n] + [torch.from_numpy(a).pin_memory().numpy() for a in arrays]
        else:
            h.load_csr(*gr.host())
            if kind != "query":
                h.levelize()
            h.sync()
        if kind == "whatif":
            e, new, old = (x.cpu().numpy() for x in gr.change(seed + 1))
            s["changes"] = [(e.astype(np.int32), new), (e.astype(np.int32), old)]
        s["out"] = [torch.empty(case["k"]).pin_memory().numpy() for _ in range(2)]
    elif kind == "batch":
        b = s["batch"] = cpg_b200.Batch()
        for i, c in enumerate(_blocks(case, 200_000)):
            b.add_graph(*_Graph(seed * 1000 + i, **c).host())
        b.commit()
        ks = _batch_ks(case)
        b.set_queries(list(range(len(ks))), ks)
        b.run(True)
        b.autotune()
        s["rebuild"], s["queries"] = case["rebuild"], len(ks)
    elif kind == "serve":
        srv = s["server"] = cpg_b200.Server()
        changes = []
        for i, c in enumerate(_blocks(case, 100_000)):
            gr = _Graph(seed * 1000 + i, **c)
            srv.add_graph(*gr.host())
            changes.append([x.cpu().numpy() for x in gr.change(seed * 1000 + i)])
        srv.start()
        s["requests"] = []
        for g, k, change in _requests(case):
            e, new, old = changes[g]
            upd = (None, None) if change is None else (e.astype(np.int32), new if change else old)
            s["requests"].append((g, k) + upd)
    elif kind == "bvss_levels":
        n, adjp, adj, _, _ = _local(case, seed)
        s["bvss"] = cpg_b200.Bvss(n, adjp, adj)
    elif kind == "bvss_pairs":
        n, adjp, adj, m, g = _local(case, seed)
        with cpg_b200.CpGen() as h:
            h.load_csr(n, adjp, adj, (0.1 + 9.9 * torch.rand(m, generator=g, device=DEV)).cpu().numpy())
            succ = h.get_sfxt()[1]
        s["bvss"] = cpg_b200.Bvss(n, adjp, adj, succ)
        pick = torch.randperm(n - case["width"], generator=g, device=DEV)[:case["sources"]]  # rows with fan-out
        s["sources"] = pick.sort()[0].int().cpu().numpy()
        s["most"] = case["sources"] * case["deg"]
    else:
        s["costs"], s["k"] = _costs(case, seed), case["k"]
        s["out"] = torch.empty(case["k"], device=DEV)
        torch.cuda.synchronize()
    return s


def _costs(case, seed):
    # path costs: a shortest path and exponentially more paths above it; a few zeros
    g = _gen(seed)
    x = 40.0 + 2.0 * torch.log1p(1000.0 * torch.rand(case["n"], generator=g, device=DEV))
    x[torch.rand(case["n"], generator=g, device=DEV) < 0.001] = 0.0
    return x


def run(s):
    kind = s["kind"]
    if kind == "query":
        h = s["handle"]
        h.reset()
        h.report_paths(s["k"])
        return h.get_slacks(s["k"], s["out"][0])
    if kind == "requery":
        h = s["handle"]
        h.report_paths(s["k"])
        return h.get_slacks(s["k"], s["out"][0])
    if kind == "whatif":
        h, got = s["handle"], []
        for (e, w), out in zip(s["changes"], s["out"]):
            h.update_delays(e, w)
            h.report_paths(s["k"])
            got.append(h.get_slacks(s["k"], out))
        return got
    if kind == "load":
        h = s["handle"]
        h.load_csr(*s["csr"])
        h.report_paths(s["k"])
        return h.get_slacks(s["k"], s["out"][0])
    if kind == "batch":
        b = s["batch"]
        b.run(s["rebuild"])
        return [b.costs(q) for q in range(s["queries"])]
    if kind == "serve":
        srv = s["server"]
        tickets = [srv.submit(g, k, e, w) for g, k, e, w in s["requests"]]
        return [srv.wait(t)[0] for t in tickets]
    if kind == "bvss_levels":
        return s["bvss"].levels()[0]
    if kind == "bvss_pairs":
        return s["bvss"].discover_pairs(s["sources"], s["most"])[0]
    got = cpg_b200.select_topk(s["costs"].data_ptr(), s["costs"].numel(), s["k"], s["out"].data_ptr())
    return s["out"][:got]


def _query_bytes(n, m, k):
    # offsets, heads and delays in; distance, successor and level of each vertex and the costs out
    return 4 * (n + 1) + 8 * m + 12 * n + 4 * k


def work(case):
    kind = case["kind"]
    if kind in ("query", "requery", "whatif", "load"):
        n, m, k = case["pins"] + 2, int(case["pins"] * case["mean"]), case["k"]
        if kind == "requery":  # the suffix tree's distances and successors in, the costs out
            return {"bytes": 8 * n + 4 * k, "flops": 3 * k}
        if kind == "whatif":
            return {"bytes": 2 * (_query_bytes(n, m, k) + 8 * (m // 100)), "flops": 4 * m}
        return {"bytes": _query_bytes(n, m, k), "flops": 2 * m}
    if kind in ("batch", "serve"):
        blocks = _blocks(case, 200_000 if kind == "batch" else 100_000)
        size = [(c["pins"] + 2, int(c["pins"] * c["mean"])) for c in blocks]
        if kind == "batch":
            per = [_query_bytes(n, m, k) if case["rebuild"] else 8 * n + 4 * k
                   for (n, m), k in zip(size, _batch_ks(case))]
        else:
            per = [8 * size[g][0] + 4 * k if change is None else
                   _query_bytes(*size[g], k) + 8 * (size[g][1] // 100)
                   for g, k, change in _requests(case)]
        return {"bytes": sum(per), "flops": 0}
    if kind == "bvss_levels":
        n = case["levels"] * case["width"]
        # a head's bit and a row id for each slice in, a level for each row out
        return {"bytes": 4 * n + n * case["deg"] * 5, "flops": 0}
    if kind == "bvss_pairs":
        pairs = case["sources"] * case["deg"]
        return {"bytes": 4 * case["sources"] + 13 * pairs, "flops": 0}
    return {"bytes": 4 * case["n"] + 4 * case["k"], "flops": 0}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("query", "requery", "load"):
        return _graph(case, seed).lowest(case["k"])
    if kind == "whatif":
        gr = _graph(case, seed)
        e, new, _ = gr.change(seed + 1)
        w = gr.w.clone()
        w[e] = new
        return [gr.lowest(case["k"], w), gr.lowest(case["k"])]
    if kind == "batch":
        return [_Graph(seed * 1000 + i, **c).lowest(k)
                for i, (c, k) in enumerate(zip(_blocks(case, 200_000), _batch_ks(case)))]
    if kind == "serve":
        graphs = [_Graph(seed * 1000 + i, **c) for i, c in enumerate(_blocks(case, 100_000))]
        most, changed, got = {}, {}, {}
        at = []
        for g, k, change in _requests(case):  # the delays each request sees, and the most paths asked of them
            changed[g] = changed.get(g, 0) if change is None else change
            at.append((g, changed[g], k))
            most[at[-1][:2]] = max(most.get(at[-1][:2], 0), k)
        for (g, new), k in most.items():
            w = graphs[g].w.clone()
            if new:
                e, fresh, _ = graphs[g].change(seed * 1000 + g)
                w[e] = fresh
            got[g, new] = graphs[g].lowest(k, w)
        return [got[g, new][:k] for g, new, k in at]
    if kind == "topk":
        x = _costs(case, seed)
        x = x[x != 0.0].double()
        return torch.sort(x)[0][:case["k"]].cpu()
    return None  # levels and pairs are whole numbers
