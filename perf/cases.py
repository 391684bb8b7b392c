"""Performance cases of lighttraffic_gb300: what its users have it do, at the sizes they do it.

Every case is one call (or one served load) through the package's entry points on a
seeded RMAT graph (a=0.57 b=0.19 c=0.19 d=0.05, the generator behind the repository's
configurations):

  ppr       Engine.ppr on a graph resident in HBM, counts to page-locked host memory
  pagerank  Engine.pagerank on a resident graph, counts to page-locked host memory
  device    lt_walk_device / lt_walk_device_compact on the caller's device buffers
            (PPR, PageRank or generic walks, with endpoints and paths where asked for)
  batch     many PPR queries in one launch: lt_ppr_batch_device, or Engine.ppr_batch
            from and to host arrays
  ooc       Engine.ppr / Engine.pagerank with a device cache smaller than the graph,
            from a cold cache as every run of the command-line programs
  serve     a burst of PPR queries through the continuous-batching server
  generate  Graph.rmat, which every benchmark and most tests start with

The random stream is keyed by walker and step, so every output is a whole number that
does not depend on the schedule; there is no rounding, hence no exact().  The order of
a sparse result's pairs inside a query is unspecified: run() sorts them by vertex, as a
program that compares or merges results does, or spreads them over a dense row per query.
"""
import ctypes
import math

import numpy as np
import torch

import lighttraffic_gb300 as lt

PPR, PAGERANK, WALK = lt.APP_PPR, lt.APP_PAGERANK, lt.APP_WALK
SOURCE, UNIFORM, PER_VERTEX = lt.START_SOURCE, lt.START_UNIFORM, lt.START_PER_VERTEX


def listed():
    return [
        # an interactive single-source query on a small graph (the size most tests use): latency
        dict(name="ppr-small", kind="ppr", scale=16, edges=1 << 20, walkers=20000, per_vertex=0, prob=0.15),
        # the small in-memory configuration: 2|V| walks from one source
        dict(name="ppr-resident", kind="ppr", scale=20, edges=1 << 24, walkers=0, per_vertex=2, prob=0.15),
        # the HBM-roofline configuration: PageRank, 2|V| walkers starting one per vertex
        dict(name="pagerank-resident", kind="pagerank", scale=23, edges=1 << 27, per_vertex=2, length=10, runs=1,
             start=PER_VERTEX),
        # raw step kernel on u64 arrays a caller keeps on the device, uniform starts, ragged sizes
        dict(name="pagerank-device-u64", kind="device", app=PAGERANK, wide=True, scale=21, edges=40000003,
             walkers=1500007, length=10, start=UNIFORM, prob=0.85, paths=False),
        # a corpus of walks for embedding training: every vertex of the walk is written out
        dict(name="walk-paths", kind="device", app=WALK, wide=False, scale=22, edges=1 << 26, walkers=4700001,
             length=10, start=PER_VERTEX, prob=0.0, paths=True),
        # fixed-length walks of the roofline configuration, endpoints only
        dict(name="walk-endpoints", kind="device", app=WALK, wide=False, scale=23, edges=1 << 27, walkers=9221596,
             length=10, start=PER_VERTEX, prob=0.0, paths=False),
        # batched multi-source PPR, the scaled batch configuration, device arrays in and out
        dict(name="batch", kind="batch", host=False, scale=22, edges=1 << 26, queries=256, median=10000, sigma=1.5,
             low=1000, high=1000000, prob=0.15),
        # a small batch from and to host arrays: latency
        dict(name="batch-small", kind="batch", host=True, scale=16, edges=1 << 20, queries=16, median=2000, sigma=0.5,
             low=1000, high=5000, prob=0.15),
        # out-of-core PPR with the learned prefetcher, the scaled out-of-core configuration
        dict(name="ooc-learned", kind="ooc", app=PPR, sched=lt.SCHED_LEARNED, scale=24, edges=1 << 28, part_kb=32768,
             partitions=16, pool=1 << 22, walkers=8388608, length=0, prob=0.15),
        # out-of-core PageRank in waves, pool large enough for every walker
        dict(name="ooc-pagerank", kind="ooc", app=PAGERANK, sched=lt.SCHED_BATCHED, scale=20, edges=1 << 24,
             part_kb=1024, partitions=24, pool=0, walkers=700001, length=10, prob=0.85),
        # a burst of queries at a server whose graph does not fit its cache
        dict(name="serve", kind="serve", scale=20, edges=1 << 24, part_kb=1024, partitions=24, pool=1 << 22,
             queries=48, median=10000, sigma=1.0, low=1000, high=100000, prob=0.15),
        # the graph of the small in-memory configuration
        dict(name="generate", kind="generate", scale=20, edges=1 << 24),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["ppr", "pagerank", "device", "device", "batch", "ooc", "serve", "generate"])
    if kind == "ppr":
        scale = rng.randint(14, 22)
        return dict(kind=kind, scale=scale, edges=_log(rng, 8 << scale, 24 << scale),
                    walkers=_log(rng, 10000, 3000000), per_vertex=0, prob=round(rng.uniform(0.1, 0.5), 2))
    if kind == "pagerank":
        scale = rng.randint(16, 22)
        return dict(kind=kind, scale=scale, edges=_log(rng, 8 << scale, 24 << scale), per_vertex=rng.choice([1, 2, 3]),
                    length=rng.randint(4, 20), runs=rng.choice([1, 1, 2]), start=rng.choice([UNIFORM, PER_VERTEX]))
    if kind == "device":
        scale = rng.randint(16, 22)
        app = rng.choice([PPR, PAGERANK, WALK, WALK])
        return dict(kind=kind, app=app, wide=rng.random() < 0.4, scale=scale, edges=_log(rng, 8 << scale, 24 << scale),
                    walkers=_log(rng, 20000, 5000000), length=0 if app == PPR else rng.randint(4, 40),
                    start=SOURCE if app == PPR else rng.choice([UNIFORM, PER_VERTEX]),
                    prob=round(rng.uniform(0.1, 0.5), 2) if app == PPR else 0.85 if app == PAGERANK else 0.0,
                    paths=app == WALK and rng.random() < 0.6)
    if kind == "batch":
        host = rng.random() < 0.4
        scale = rng.randint(14, 16) if host else rng.randint(16, 22)
        return dict(kind=kind, host=host, scale=scale, edges=_log(rng, 8 << scale, 16 << scale),
                    queries=_log(rng, 3, 24 if host else 400), median=_log(rng, 1000, 10000), sigma=round(rng.uniform(0.3, 1.5), 2),
                    low=rng.choice([1, 100, 1000]), high=10000 if host else _log(rng, 20000, 300000),
                    prob=round(rng.uniform(0.1, 0.4), 2))
    if kind == "ooc":
        scale = rng.randint(18, 22)
        app = rng.choice([PPR, PPR, PAGERANK])
        return dict(kind=kind, app=app, sched=rng.choice([lt.SCHED_LEARNED, lt.SCHED_FREQUENCY, lt.SCHED_BATCHED]),
                    scale=scale, edges=_log(rng, 12 << scale, 16 << scale), part_kb=1024 << scale >> 20,
                    partitions=rng.randint(12, 24), pool=rng.choice([0, 1 << 20]),
                    walkers=_log(rng, 100000, 2000000 if app == PPR else 700000), length=0 if app == PPR else rng.randint(4, 10),
                    prob=0.15 if app == PPR else 0.85)
    if kind == "serve":
        scale = rng.randint(18, 20)
        return dict(kind=kind, scale=scale, edges=_log(rng, 12 << scale, 16 << scale), part_kb=1024 << scale >> 20,
                    partitions=rng.randint(12, 24), pool=1 << 22, queries=_log(rng, 4, 60), median=_log(rng, 2000, 10000),
                    sigma=round(rng.uniform(0.3, 1.0), 2), low=1000, high=100000, prob=round(rng.uniform(0.1, 0.3), 2))
    scale = rng.randint(14, 20)
    return dict(kind=kind, scale=scale, edges=_log(rng, 4 << scale, 16 << scale))


def _walkers(c):
    """Lognormal walk counts of the case's queries (the same for every seed)."""
    w = np.exp(np.random.default_rng(1).normal(math.log(c["median"]), c["sigma"], c["queries"]))
    return np.clip(np.round(w), c["low"], c["high"]).astype(np.uint64)


def _queries(c, seed, rowptr):
    """Zipf sources over the out-degree rank, walk counts, keys."""
    rng = np.random.default_rng(seed)
    deg = np.diff(rowptr.astype(np.int64))
    order = np.argsort(-deg, kind="stable")
    p = np.arange(1, len(deg) + 1, dtype=np.float64) ** -1.1
    src = order[rng.choice(len(deg), size=c["queries"], p=p / p.sum())].astype(np.uint32)
    return src, _walkers(c), rng.integers(1, 1 << 62, c["queries"]).astype(np.uint64)


def _graph(c, part_bytes=32 << 20, seed=1):
    return lt.Graph.rmat(c["scale"], c["edges"], seed=seed, part_bytes=part_bytes)


def prepare(case, seed):
    c, k = case, case["kind"]
    s = dict(case=c, seed=seed)
    if k == "generate":
        s["rowptr"] = np.zeros((1 << c["scale"]) + 1, np.int64)
        return s
    if k in ("ooc", "serve"):
        g = _graph(c, c["part_kb"] << 10)
        e = lt.Engine(g, partitions=c["partitions"], batch=c["pool"], seed=seed, sched=c.get("sched", lt.SCHED_LEARNED))
        s.update(graph=g, engine=e)
        if k == "ooc":
            s["out"] = lt.pinned_empty(g.num_nodes)
            return s
        rng = np.random.default_rng(seed)
        n, w = c["queries"], _walkers(c).tolist()
        s.update(sources=rng.integers(0, g.num_nodes, n).tolist(), walkers=w, seeds=rng.integers(1, 1 << 62, n).tolist(),
                 pairs=_Pairs(n, g.num_nodes, sum(w)),
                 server=lt.Server(e, max_active=64, table_slots=1 << 24, prob=c["prob"]))
        return s
    g = _graph(c)
    if k in ("ppr", "pagerank"):
        s.update(graph=g, engine=lt.Engine(g, seed=seed), out=lt.pinned_empty(g.num_nodes),
                 walkers=int(c["per_vertex"] * g.num_nodes) or c["walkers"])
        return s
    if k == "batch":
        src, w, sd = _queries(c, seed, g.csr_views()[0])
        s.update(graph=g, engine=lt.Engine(g, seed=seed), sources=src, walkers=w, seeds=sd)
        n, total = len(src), int(w.sum())
        if c["host"]:
            s["out"] = (lt.pinned_empty(n + 1, np.uint64), lt.pinned_empty(total, np.uint32), lt.pinned_empty(total, np.uint32))
            s["dense"] = np.zeros((n, g.num_nodes), np.int32)
        else:
            s["dev"] = [torch.from_numpy(x).cuda() for x in (src.view(np.int32), w.view(np.int64), sd.view(np.int64))]
            s["out"] = (torch.zeros(n + 1, dtype=torch.int64, device="cuda"), torch.zeros(total, dtype=torch.int32, device="cuda"),
                        torch.zeros(total, dtype=torch.int32, device="cuda"))
            s["pairs"] = _Pairs(n, g.num_nodes, total)
        s["total"] = total
        return s
    # caller's device buffers
    rp, col = g.csr_views()
    V, W = g.num_nodes, c["walkers"]
    d_rp = torch.from_numpy(rp.view(np.int64)).cuda()
    s.update(V=V, col=torch.from_numpy(col.view(np.int32)).cuda(),
             scratch=torch.zeros(max(1, lt.lib.lt_walk_scratch_bytes() // 8), dtype=torch.int64, device="cuda"))
    if c["wide"]:
        s["rows"] = d_rp
    else:
        s["rows"] = torch.empty(V + 1, dtype=torch.int32, device="cuda")
        lt.check(lt.lib.lt_rowptr_narrow(d_rp.data_ptr(), s["rows"].data_ptr(), V, torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
    s["counts"] = None if c["app"] == WALK else torch.zeros(V, dtype=torch.int64 if c["wide"] else torch.int32, device="cuda")
    s["endpoints"] = torch.zeros(W, dtype=torch.int32, device="cuda") if c["app"] == WALK else None
    s["paths"] = torch.zeros(W * (c["length"] + 1), dtype=torch.int32, device="cuda") if c["paths"] else None
    return s


class _Pairs:
    """Sparse results in canonical form on the device: query * V + vertex in ascending order and the counts, in
    buffers of the batch's capacity (-1 and 0 behind the last pair)."""

    def __init__(self, n, V, total):
        self.first = torch.arange(n, device="cuda", dtype=torch.int32 if n * V < 1 << 31 else torch.int64) * V
        self.key = torch.empty(total, dtype=self.first.dtype, device="cuda")
        self.count = torch.empty(total, dtype=torch.int32, device="cuda")

    def __call__(self, off, vertices, counts):
        k = vertices.numel()
        key = torch.repeat_interleave(self.first, off[1:] - off[:-1], output_size=k) + vertices
        self.key[k:] = -1
        self.count[k:] = 0
        self.key[:k], at = torch.sort(key)
        torch.index_select(counts, 0, at, out=self.count[:k])
        return off, self.key, self.count


class _GraphView(np.ndarray):
    """An array in a graph's host memory; keeps the graph open."""


def _ptr(t):
    return None if t is None else t.data_ptr()


def run(state):
    s = state
    c, k = s["case"], s["case"]["kind"]
    if k == "ppr":
        return s["engine"].ppr(0, s["walkers"], c["prob"], out=s["out"]).view(np.int64)
    if k == "pagerank":
        return s["engine"].pagerank(s["walkers"], length=c["length"], runs=c["runs"], start=c["start"], out=s["out"]).view(np.int64)
    if k == "device":
        if s["counts"] is not None:
            s["counts"].zero_()
        call = lt.lib.lt_walk_device if c["wide"] else lt.lib.lt_walk_device_compact
        lt.check(call(c["app"], c["start"], _ptr(s["rows"]), _ptr(s["col"]), s["V"], 0, c["walkers"], c["length"],
                      ctypes.c_float(c["prob"]), 0, s["seed"], _ptr(s["counts"]), _ptr(s["endpoints"]), _ptr(s["paths"]),
                      _ptr(s["scratch"]), None, torch.cuda.current_stream().cuda_stream))
        return [t for t in (s["counts"], s["endpoints"], s["paths"]) if t is not None]
    if k == "batch":
        off, v, n = *s["out"][:2], len(s["sources"])
        if c["host"]:
            off, v, cnt = s["engine"].ppr_batch(s["sources"], s["walkers"], s["seeds"], c["prob"], out=s["out"])
            dense = s["dense"]
            dense.fill(0)
            for q, (a, b) in enumerate(zip(off[:-1].tolist(), off[1:].tolist())):
                dense[q, v[a:b]] = cnt[a:b]
            return off.view(np.int64), dense
        src, w, sd = s["dev"]
        lt.check(lt.lib.lt_ppr_batch_device(s["engine"]._h, n, _ptr(src), _ptr(w), _ptr(sd), ctypes.c_float(c["prob"]), _ptr(off), _ptr(v),
                                            _ptr(s["out"][2]), s["total"], torch.cuda.current_stream().cuda_stream))
        pairs = int(off[n])
        return s["pairs"](off, v[:pairs], s["out"][2][:pairs])
    if k == "ooc":
        e = s["engine"]
        e.drop_cache()
        if c["app"] == PPR:
            return e.ppr(0, c["walkers"], c["prob"], out=s["out"]).view(np.int64)
        return e.pagerank(c["walkers"], length=c["length"], start=PER_VERTEX, alpha=c["prob"], out=s["out"]).view(np.int64)
    if k == "serve":
        return _serve(s)
    g = _graph(c, seed=s["seed"])
    rp, col = g.csr_views()
    V = g.num_nodes
    s["rowptr"][:V + 1] = rp.view(np.int64)
    s["rowptr"][V + 1:] = c["edges"]
    col = col.view(np.int32).view(_GraphView)
    col.graph = g
    return V, s["rowptr"], col


def _serve(s):
    srv = s["server"]
    order = {srv.submit(a, w, sd): i for i, (a, w, sd) in enumerate(zip(s["sources"], s["walkers"], s["seeds"]))}
    res, left = [None] * len(order), len(order)
    done, n, ms = ctypes.c_int(), ctypes.c_uint64(), ctypes.c_double()
    u32p = ctypes.POINTER(ctypes.c_uint32)
    while left:
        srv.step()
        for t in srv.finished(len(order)):
            cap = s["walkers"][order[t]]
            v, cnt = np.empty(cap, np.uint32), np.empty(cap, np.uint32)
            lt.check(lt.lib.lt_serve_result(srv._h, t, ctypes.byref(done), ctypes.byref(n), v.ctypes.data_as(u32p), cnt.ctypes.data_as(u32p),
                                            cap, ctypes.byref(ms)))
            res[order[t]] = (v[:n.value], cnt[:n.value])
            left -= 1
    off = np.zeros(len(res) + 1, np.int64)
    np.cumsum([len(v) for v, _ in res], out=off[1:])
    dev = [torch.from_numpy(np.concatenate([r[i] for r in res]).view(np.int32)).cuda() for i in (0, 1)]
    return s["pairs"](torch.from_numpy(off).cuda(), *dev)


def work(case):
    """Bytes a pass cannot do without: the graph's column entries and row offsets that the hops read, each at most
    once, at 4 bytes, and the outputs.  An RMAT graph at these densities keeps about 0.55 of its 2^scale vertices."""
    c, k = case, case["kind"]
    V, E = 0.55 * (1 << c["scale"]), c["edges"]
    if k == "generate":
        return {"bytes": 4 * E + 8 * V, "flops": 0}
    mean = lambda: min(max(c["median"] * math.exp(c["sigma"] ** 2 / 2), c["low"]), c["high"])  # noqa: E731
    W = c["queries"] * mean() if "queries" in c else c.get("per_vertex", 0) * V or c["walkers"]
    hops = W * (c["length"] * c.get("runs", 1) if c.get("length") else 1 / c["prob"])
    read = 4 * min(E, hops) + 4 * min(V, 2 * hops)
    if k in ("batch", "serve"):
        return {"bytes": read + 20 * c["queries"] + 8 * min(W / 2, c["queries"] * V), "flops": 0}
    out = 8 * V
    if k == "device":
        out = 4 * W * (1 + (c["length"] + 1 if c["paths"] else 0)) if c["app"] == WALK else (8 if c["wide"] else 4) * V
    return {"bytes": read + out, "flops": 0}
