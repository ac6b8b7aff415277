"""The work this framework is used for, as cases that can be timed.

A case is one query (or one batch of queries) through the Python interface:
`Context.amhj`, `Context.lftj`, `Batch.run`.  Every pass returns what the
call returns to its user: the result's count and its order-independent 64-bit
tuple checksum as two 64-bit words, and the result's columns where the query
asks for its tuples.

Inputs are drawn on the GPU from the seed: uniform and Zipf int32 key columns
(with a rank-to-key permutation, so that frequent keys are spread over the
key range) and R-MAT edge relations (self-loops and repeated edges dropped,
edges oriented from the lower to the higher id, rows shuffled), the shapes
of `accmultiwayjoins_b200.data`.  Out-of-core relations are in pinned host
memory.
"""
import math

import numpy as np
import torch

from accmultiwayjoins_b200 import Context, data

DEV = "cuda"
M64 = (1 << 64) - 1

# R-MAT skews: of the triangle workload and of the skewed 4-clique
RMAT_TRI = (0.57, 0.19, 0.19)
RMAT_SKEW = (0.6, 0.15, 0.15)


def listed():
    return [
        # the smallest call: a 3-way chain of 10K-row relations, the size at
        # which launches, allocations and waits on the host decide the latency
        {"name": "chain_10k", "kind": "chain", "rels": 3, "rows": 10_000, "domain": 4_096, "theta": 0.0, "ws": 0,
         "fib": 0},
        # the plain 3-way chain of the headline configuration: 1M rows each,
        # keys uniform in [0, 2^18)
        {"name": "chain_1m", "kind": "chain", "rels": 3, "rows": 1_000_000, "domain": 1 << 18, "theta": 0.0, "ws": 0,
         "fib": 0},
        # a skewed 4-way chain at an odd size, with work sharing and
        # frequent-item buffering on, as the switches are meant to be used
        {"name": "chain_zipf", "kind": "chain", "rels": 4, "rows": 1_300_003, "domain": 1_048_577, "theta": 1.0,
         "ws": 1, "fib": 1},
        # the 4-way star of the headline configuration: 60M fact rows of Zipf
        # foreign keys into four dimensions (the largest input of a hash join)
        {"name": "star_60m", "kind": "star", "rows": 60_000_000, "dims": 4, "dim_rows": 1_000_000, "theta": 1.1,
         "rows_out": False},
        # a star whose tuples the caller wants, as host columns
        {"name": "star_rows_1m", "kind": "star", "rows": 1_000_003, "dims": 3, "dim_rows": 200_000, "theta": 1.1,
         "rows_out": True},
        # triangles of a small graph by the leapfrog triejoin: latency again
        {"name": "tri_64k", "kind": "triangle", "edges": 1 << 16, "scale": 13, "op": "dfs"},
        # triangles of the headline graph (R-MAT scale 20, 16M edges), depth first
        {"name": "tri_16m", "kind": "triangle", "edges": 1 << 24, "scale": 20, "op": "dfs"},
        # triangles breadth first, at a middle size
        {"name": "tri_bfs_2m", "kind": "triangle", "edges": 2_000_001, "scale": 17, "op": "bfs"},
        # R(a,b) S(b,c) T(a,c) over three different relations
        {"name": "tri_rst_1m", "kind": "triangle", "edges": 1 << 20, "scale": 16, "op": "rst"},
        # the skewed 4-clique of the headline configuration through the hash
        # join's FOUR query with work sharing and frequent-item buffering
        # (the longest single query)
        {"name": "four_64m", "kind": "four", "edges": 1 << 26, "scale": 22},
        # many uneven queries (chains, stars, triangles) in one replayed batch
        {"name": "batch_128", "kind": "batch", "queries": 128, "max_rows": 1_000_000, "mix": 4},
        # a 4-way chain larger than its memory budget, every relation in host
        # memory: the staged out-of-core join
        {"name": "ooc_16m", "kind": "ooc", "rels": 4, "rows": 1 << 24, "domain": 1 << 24, "budget_mb": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "chain", "chain", "star", "star", "triangle", "triangle", "triangle", "four", "batch",
                       "ooc"])
    if kind == "chain":
        rels = rng.randint(2, 5)
        rows = _log_int(rng, 10_000, 4_000_000)
        # matches per row and join, the output at most 2^25 tuples
        most = min(4.0, (2.0**25 / rows) ** (1.0 / (rels - 1)))
        domain = max(64, int(rows / rng.uniform(0.5, most)))
        theta = rng.choice([0.0, 0.0, rng.uniform(0.5, 1.2)])
        ws = rng.choice([0, 1])
        return {"kind": kind, "rels": rels, "rows": rows, "domain": domain, "theta": theta, "ws": ws,
                "fib": ws * rng.choice([0, 1])}
    if kind == "star":
        out = rng.choice([False, False, True])
        rows = _log_int(rng, 10_000, 4_000_000 if out else 60_000_000)
        return {"kind": kind, "rows": rows, "dims": rng.randint(1, 4),
                "dim_rows": min(1_000_000, _log_int(rng, 1_000, max(1_000, rows))),
                "theta": rng.choice([0.0, rng.uniform(0.5, 1.5)]), "rows_out": out}
    if kind == "triangle":
        op = rng.choice(["dfs", "dfs", "bfs", "rst", "hash"])
        edges = _log_int(rng, 10_000, {"dfs": 1 << 24, "hash": 1 << 24, "bfs": 1 << 22, "rst": 1 << 21}[op])
        return {"kind": kind, "edges": edges, "scale": max(8, round(math.log2(edges / rng.uniform(8, 20)))), "op": op}
    if kind == "four":
        edges = _log_int(rng, 1 << 14, 1 << 24)
        return {"kind": kind, "edges": edges, "scale": max(8, round(math.log2(edges / 16)))}
    if kind == "batch":
        return {"kind": kind, "queries": rng.randint(8, 128), "max_rows": _log_int(rng, 50_000, 1_000_000),
                "mix": rng.randint(1, 1 << 20)}
    rows = _log_int(rng, 1 << 20, 1 << 24)
    return {"kind": kind, "rels": rng.randint(2, 4), "rows": rows, "domain": int(rows * rng.uniform(0.7, 1.5)),
            "budget_mb": rng.choice([64, 128, 256])}


# ---- inputs ----

class _Gen:
    """The generators that the workload builders of `data` take, on the GPU,
    every column from a random stream of its own."""

    def __init__(self, seed, device=DEV):
        self.seed, self.device = seed, device

    def _rng(self, *key):
        h = 0x9E3779B97F4A7C15
        for v in (self.seed,) + key:
            h = ((h ^ int(v)) * 0xBF58476D1CE4E5B9 + 0x94D049BB133111EB) & M64
            h ^= h >> 29
        return torch.Generator(device=self.device).manual_seed(h >> 1)

    def uniform(self, n, lo, hi, seed, stream=0):
        return torch.randint(lo, hi, (n,), dtype=torch.int32, device=self.device, generator=self._rng(1, seed, stream))

    def permutation(self, n, seed, stream=0):
        return torch.randperm(n, dtype=torch.int32, device=self.device, generator=self._rng(2, seed, stream))

    def zipf(self, n, domain, theta, seed, stream=0, rank_to_key=None):
        cdf = torch.arange(1, domain + 1, dtype=torch.float64, device=self.device).pow_(-theta).cumsum_(0)
        x = torch.rand(n, dtype=torch.float64, device=self.device, generator=self._rng(3, seed, stream)) * cdf[-1]
        rank = torch.searchsorted(cdf, x).clamp_(max=domain - 1)
        return rank_to_key[rank] if rank_to_key is not None else rank.to(torch.int32)

    def rmat(self, scale, nedges, a, b, c, seed):
        g = self._rng(4, seed)
        u = torch.zeros(nedges, dtype=torch.int64, device=self.device)
        v = torch.zeros_like(u)
        for _ in range(scale):
            x = torch.rand(nedges, device=self.device, generator=g)
            low = x >= a + b
            u = 2 * u + low
            v = 2 * v + (((x >= a) & ~low) | (x >= a + b + c))
        key = torch.minimum(u, v) << 32 | torch.maximum(u, v)
        key = torch.unique(key[u != v])
        key = key[torch.randperm(key.numel(), device=self.device, generator=g)]
        return (key >> 32).to(torch.int32), key.to(torch.int32)


class _Sizes:
    """Columns of the same lengths without contents."""

    def uniform(self, n, *a, **k):
        return torch.empty(n, dtype=torch.int32, device="meta")

    permutation = zipf = uniform

    def rmat(self, scale, nedges, *a, **k):
        return self.uniform(nedges), self.uniform(nedges)


def _dim_sizes(case):
    """The dimensions shrink from the largest one, as in the 4-way star (1M, 200K, 100K, 10K rows)."""
    return [max(64, case["dim_rows"] * s // 100) for s in (100, 20, 10, 1)[:case["dims"]]]


def _queries(case, gen):
    """The case's queries: (query type, [(columns, attributes)]) each."""
    kind = case["kind"]
    if kind in ("chain", "ooc"):
        n, m, theta = case["rows"], case["domain"], case.get("theta", 0.0)
        rels = data.chain_relations(n, m, case["rels"], seed=1, gen=gen)
        if theta:
            # skewed build sides: the join column of every relation but the first
            for i in range(1, case["rels"]):
                rels[i][0][0] = gen.zipf(n, m, theta, 1 + i, 7, rank_to_key=gen.permutation(m, 1 + i, 8))
        return [("NORMAL", rels)]
    if kind == "star":
        fact, dims = data.star_relations(case["rows"], _dim_sizes(case), case["theta"], seed=3, gen=gen)
        return [("NORMAL", [fact] + dims)]
    if kind == "batch":
        return [(q["qt"], q["rels"]) for q in data.query_mix(case["queries"], seed=case["mix"],
                                                             max_rows=case["max_rows"], gen=gen)]
    if kind == "four":
        return [("FOUR", [(list(gen.rmat(case["scale"], case["edges"], *RMAT_SKEW, 22)), [0, 1])])]
    pairs = [[0, 1], [1, 2], [0, 2]] if case["op"] == "rst" else [[0, 1]]
    return [("TRI", [(list(gen.rmat(case["scale"], case["edges"], *RMAT_TRI, 20 + i)), p)
                     for i, p in enumerate(pairs)])]


def prepare(case, seed):
    queries = _queries(case, _Gen(seed))
    ooc = case["kind"] == "ooc"
    ctx = Context(0, mem_budget=case["budget_mb"] << 20) if ooc else Context(0)
    if ooc:
        host = []
        for cols, attrs in queries[0][1]:
            pinned = [torch.empty(c.shape, dtype=c.dtype, pin_memory=True) for c in cols]
            for p, c in zip(pinned, cols):
                p.copy_(c)
            host.append((pinned, attrs))
        rels = [[ctx.relation([p.numpy() for p in cols], attrs, streamed=True) for cols, attrs in host]]
        queries = [("NORMAL", host)]   # keeps the pinned memory
    else:
        rels = [[ctx.relation([c.contiguous() for c in cols], attrs) for cols, attrs in rs] for _, rs in queries]
    state = {"case": case, "ctx": ctx, "rels": rels, "inputs": queries}
    if case["kind"] == "batch":
        state["batch"] = ctx.batch()
        for (qt, _), rs in zip(queries, rels):
            state["batch"].submit(qt, rs)
    torch.cuda.synchronize()   # the relations are read on the context's own stream
    return state


def _words(*values):
    """Unsigned 64-bit results as signed words."""
    return np.array([v & M64 for v in values], dtype=np.uint64).view(np.int64)


def run(state):
    case, ctx, rels = state["case"], state["ctx"], state["rels"][0]
    kind = case["kind"]
    if kind == "batch":
        r = state["batch"].run(use_graph=True)
        return _words(*r.counts), _words(*r.checksums)
    if kind == "chain":
        r = ctx.amhj("NORMAL", rels, ws=case["ws"], fib=case["fib"])
    elif kind == "star":
        r = ctx.amhj("NORMAL", rels, materialize=case["rows_out"])
        if case["rows_out"]:
            return _words(r.count, r.checksum), r.columns
    elif kind == "four":
        r = ctx.amhj("FOUR", rels, ws=1, fib=1)
    elif kind == "ooc":
        r = ctx.amhj("NORMAL", rels, ooc=1)
    elif case["op"] == "hash":
        r = ctx.amhj("TRI", rels)
    else:
        r = ctx.lftj(rels, algo="BFS" if case["op"] == "bfs" else "DFS")
    return _words(r.count, r.checksum)


def work(case):
    """Every relation read once; two words for every query and its tuples, where asked for, written once."""
    queries = _queries(case, _Sizes())
    read = sum(4 * c.numel() for _, rels in queries for cols, _ in rels for c in cols)
    written = 16 * len(queries)
    if case.get("rows_out"):   # foreign keys: one tuple for every fact row
        written += 4 * case["rows"] * 2 * case["dims"]
    return {"bytes": float(read + written), "flops": 0.0}


# ---- the same results from plain torch, in 64 bits ----

def _mix64(z):
    for s, m in ((30, 0xBF58476D1CE4E5B9), (27, 0x94D049BB133111EB)):
        z = (z ^ ((z >> s) & ((1 << (64 - s)) - 1))) * (m - (1 << 64))
    return z ^ ((z >> 31) & ((1 << 33) - 1))


def _result(cols):
    """(count, checksum) of tuples given as columns, and the columns."""
    h = torch.full_like(cols[0], 0x9E3779B97F4A7C15 - (1 << 64), dtype=torch.int64)
    for c in cols:
        h = _mix64(h ^ (c.to(torch.int64) & 0xFFFFFFFF))
    return len(h), int(h.sum()) & M64


def _join(cols, probe, build_keys, build_payload):
    """cols extended by the payload of every match of column `probe`, in the order of the rows."""
    keys, at = torch.sort(build_keys, stable=True)
    lo, hi = torch.searchsorted(keys, cols[probe]), torch.searchsorted(keys, cols[probe], right=True)
    n = hi - lo
    row = torch.repeat_interleave(torch.arange(len(n), device=n.device), n)
    first = torch.cumsum(n, 0) - n
    match = at[lo[row] + torch.arange(len(row), device=n.device) - first[row]]
    return [c[row] for c in cols] + [build_payload[match]]


def _triangles(s, d):
    """The triangles of an oriented edge relation, from the wedges of its degree order; None where they are too many."""
    nv = int(d.max()) + 1
    deg = torch.bincount(torch.cat([s, d]).to(torch.int64), minlength=nv)
    rank = torch.empty_like(deg)
    rank[torch.argsort(deg, stable=True)] = torch.arange(nv, device=deg.device)
    a, b = rank[s.to(torch.int64)], rank[d.to(torch.int64)]
    key = torch.sort(torch.minimum(a, b) << 32 | torch.maximum(a, b))[0]
    a, b = key >> 32, key & 0xFFFFFFFF
    end = torch.searchsorted(a, a, right=True)
    n = end - torch.arange(len(a), device=a.device) - 1   # the children of a after b
    if int(n.sum()) > 1 << 27:
        return None
    row = torch.repeat_interleave(torch.arange(len(a), device=a.device), n)
    c = b[row + 1 + torch.arange(len(row), device=a.device) - (torch.cumsum(n, 0) - n)[row]]
    want = b[row] << 32 | c
    at = torch.searchsorted(key, want).clamp_(max=len(key) - 1)
    hit = key[at] == want
    back = torch.argsort(rank)
    return list(torch.sort(torch.stack([back[a[row[hit]]], back[b[row[hit]]], back[c[hit]]]), dim=0)[0].unbind(0))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("four", "batch") or case.get("op") == "rst" or case.get("rows", 0) > 1 << 25:
        return None
    (_, rels), = _queries(case, _Gen(seed))
    if kind == "triangle":
        cols = _triangles(*rels[0][0])
        return None if cols is None else _words(*_result(cols))
    cols = list(rels[0][0])
    for j, ((keys, payload), attrs) in enumerate(rels[1:]):
        cols = _join(cols, attrs[0], keys, payload)
    if case.get("rows_out"):
        return _words(*_result(cols)), [c.cpu().numpy() for c in cols]
    return _words(*_result(cols))
