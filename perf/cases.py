"""The calls that a program using gem_b200 spends its time in, as cases that can be timed and compared.

A data graph is loaded once and stays resident (one Context per graph and option set, shared by the states of a
case, as a program would keep it); every state brings new random-walk queries, drawn from the seed.  `skew` graphs
are R-MAT with the benchmark's quadrant probabilities (hubs, as in social and web graphs); the others have equal
quadrants (near-equal degrees, as in protein or molecule networks), where queries of up to 32 vertices have few
enough embeddings to be counted exactly.  All outputs are whole numbers and are compared bit for bit."""
import time

import numpy as np

import gem_b200 as gem

BUDGET = 24 << 30      # device bytes of one context: three of them fit a card beside anything else
CAP_MS = 20000         # per-call device time cap: a bound, far above every case's time
ROOM = 1 << 17         # embeddings that the enumerating program has room for
MIX = (4, 8, 12, 16, 24, 32)  # query sizes of the mixed batches (the benchmark's)


def _case(name, call, scale, ef, labels, zipf, skew, k, queries, **more):
    c = dict(name=name, call=call, scale=scale, edge_factor=ef, labels=labels, zipf=zipf, skew=skew, k=k,
             queries=queries, vertices=1 << scale)
    c.update(more)
    return c


def listed():
    return [
        # one query on a graph that fits a corner of L2: launch latency and synchronisations
        _case("plain-4k", "run", 12, 8, 4, 0.0, True, 4, 1),
        # the benchmark's small configuration, one query per call: interactive use
        _case("plain-64k", "run", 16, 8, 8, 0.0, True, 4, 4),
        # the in-core configuration's graph, one query per call
        _case("plain-4m", "run", 22, 16, 16, 1.0, True, 4, 4),
        # the small configuration as one batch of 100
        _case("batch-64k", "batch", 16, 8, 8, 0.0, True, 4, 100),
        # a batch of small queries on the scale-22 graph (heavy hubs)
        _case("batch-4m", "batch", 22, 16, 16, 1.0, True, 4, 100),
        # queries of 4 to 32 vertices in one batch: thousands of filter rows and edge tables in a wave
        _case("mixed-1m", "batch", 20, 8, 32, 0.0, False, 0, 180),
        # counts with the embedding hash: every embedding is enumerated
        _case("hash-16k", "hash", 14, 8, 16, 0.0, True, 4, 16),
        # embeddings listed, not just counted
        _case("enumerate-16k", "enumerate", 14, 8, 8, 0.0, False, 4, 1),
        # adjacency in pinned host memory, streamed through the device
        _case("out-of-core-1m", "batch", 20, 16, 16, 1.0, True, 4, 50, ooc=True),
        # relaxed matching (-t 1) of a query with a cycle
        _case("relaxed-64k", "relaxed", 16, 8, 8, 0.0, True, 5, 1, threshold=1),
        # candidate lists alone, slack 1, on a graph of ragged size
        _case("filter-1m", "filter", 20, 16, 23, 1.0, True, 8, 1, threshold=1, vertices=1000003),
        # a burst of requests to the server
        _case("serve-64k", "serve", 16, 8, 8, 0.0, True, 4, 100),
    ]


def draw(rng):
    call = rng.choice(("run", "run", "batch", "mixed", "mixed", "hash", "enumerate", "ooc", "relaxed", "filter", "serve"))
    lo, hi = {"run": (10, 21), "batch": (11, 19), "mixed": (11, 20), "hash": (10, 14), "enumerate": (11, 15),
              "ooc": (14, 20), "relaxed": (10, 16), "filter": (11, 20), "serve": (11, 17)}[call]
    scale = rng.randint(lo, hi)
    ef = rng.randint(4, 16)
    zipf = rng.choice((0.0, 1.0))
    labels = rng.randint(8, 20) if zipf == 0.0 else rng.randint(16, 48)
    skew, k, queries, more = True, rng.choice((3, 4, 4)), rng.randint(1, 4), {}
    # any number of vertices, not just powers of two
    more["vertices"] = (1 << scale) - (rng.randint(0, 1 << (scale - 2)) if rng.random() < 0.7 else 0)
    if call in ("batch", "ooc", "serve"):
        queries = int(5 * 2 ** rng.uniform(0, 4.6))
    if call == "mixed":  # up to 32 vertices; labels enough that the counts stay bounded, above 64 too
        skew, zipf, k, ef, labels = False, 0.0, 0, rng.randint(3, 8), rng.randint(24, 90)
        queries = int(7 * 2 ** rng.uniform(0, 4.4))
        more["largest"] = rng.choice((12, 16, 24, 32))
    if call == "hash":
        queries, zipf, labels = rng.randint(1, 16), 0.0, rng.randint(16, 24)
        more["index"] = rng.choice(("auto", "cuckoo"))
    if call == "enumerate":
        skew, k, queries, zipf, labels, ef = False, rng.choice((3, 4, 5)), 1, 0.0, rng.randint(7, 12), rng.randint(4, 8)
    if call == "ooc":
        more["ooc"] = True
    if call == "relaxed":
        k, queries, zipf, labels, more["threshold"] = 5, 1, 0.0, rng.randint(8, 16), 1
    if call == "filter":
        k, queries, more["threshold"] = rng.randint(3, 32), 1, rng.choice((0, 1, 2))
        labels = rng.randint(3, 90)
    call = {"mixed": "batch", "ooc": "batch"}.get(call, call)
    c = _case("", call, scale, ef, labels, zipf, skew, k, queries, **more)
    del c["name"]
    return c


def _graph(case):
    p = (0.57, 0.19, 0.19) if case["skew"] else (0.25, 0.25, 0.25)
    seed = 0x47454D00 + case["scale"]
    g = gem.HostGraph.rmat(case["scale"], case["edge_factor"], *p, seed=seed)
    n = case["vertices"]
    if n != 1 << case["scale"]:  # the subgraph induced by the first n vertices
        off, nbr, lab = g.arrays()
        nbr = nbr[:int(off[n])]
        keep = nbr < n
        at = np.zeros(len(nbr) + 1, np.uint64)
        np.cumsum(keep, out=at[1:])
        g = gem.HostGraph.from_csr(at[off[:n + 1]], nbr[keep], lab[:n])
    return g.set_labels(case["labels"], case["zipf"], seed=seed ^ 0x4C)


_resident = {}  # the graph in use: {key: (host graph, context)}, one entry


def _context(case):
    key = tuple(case.get(f) for f in ("scale", "edge_factor", "skew", "vertices", "labels", "zipf", "ooc", "index")) + (
        case["call"] == "serve",)
    if key not in _resident:
        _resident.clear()
        g = _graph(case)
        ctx = gem.Context(time_cap_ms=CAP_MS, budget_bytes=BUDGET, ooc=bool(case.get("ooc")),
                          index_kind=gem.IDX_CUCKOO if case.get("index") == "cuckoo" else gem.IDX_AUTO)
        ctx.load_graph(g)
        _resident[key] = (g, ctx)
    return _resident[key]


def prepare(case, seed):
    g, ctx = _context(case)
    n, k = case["queries"], case["k"]
    seed = (seed + 1) * 0x9E3779B1 % (1 << 40)
    if k == 0:
        sizes = [s for s in MIX if s <= case.get("largest", 32)]
        per = [n // len(sizes) + (i < n % len(sizes)) for i in range(len(sizes))]
        qs = [q for i, s in enumerate(sizes) if per[i] for q in gem.gen_queries(g, s, gem.ANY, per[i], seed=seed + s)]
    elif case["call"] == "relaxed":  # a query with a cycle (a tree has nothing to remove)
        qs = gem.gen_queries(g, k, gem.ANY, 64, seed=seed)
        qs = ([q for q in qs if q.ne == k] or sorted(qs, key=lambda q: -q.ne))[:n]
    else:
        qs = gem.gen_queries(g, k, gem.ANY, n, seed=seed)
    st = {"ctx": ctx, "call": case["call"], "queries": qs, "threshold": case.get("threshold", 0)}
    if case["call"] == "enumerate":  # a program that lists embeddings has room for so many: a query that fits
        st["room"] = ROOM
        st["queries"] = [next(q for q in gem.gen_queries(g, k, gem.ANY, 32, seed=seed) if ctx.run(q)["count"] <= ROOM)]
    if case["call"] == "filter":  # no list is longer than its label's vertices
        st["room"] = k * int(np.bincount(g.arrays()[2]).max())
    return st


def _serve(ctx, queries):
    """Submits every query and collects the answers as they come (a busy server takes the query later)."""
    counts = np.zeros(len(queries), np.uint64)
    status = np.zeros(len(queries), np.int32)
    todo, open_ = list(range(len(queries)))[::-1], []
    while todo or open_:
        while todo:
            t = ctx.submit(queries[todo[-1]])
            if t is None:
                break
            open_.append((todo.pop(), t))
        still = []
        for i, t in open_:
            r = ctx.poll(t)
            if r is None:
                still.append((i, t))
            else:
                counts[i], status[i] = r["count"], r["status_code"]
        if len(still) == len(open_):
            time.sleep(2e-5)
        open_ = still
    return {"counts": counts, "status": status}


def run(state):
    ctx, qs, call = state["ctx"], state["queries"], state["call"]
    if call == "run":
        return {"counts": np.array([ctx.run(q)["count"] for q in qs], np.uint64)}
    if call == "batch":
        st, counts, status = ctx.batch_counts(qs)
        return {"counts": counts, "status": status}
    if call == "hash":
        st, rs = ctx.batch(qs, mode=gem.MODE_HASH)
        return {"counts": np.array([r["count"] for r in rs], np.uint64),
                "hashes": np.array([r["emb_hash"] for r in rs], np.uint64),
                "status": np.array([r["status_code"] for r in rs], np.int32)}
    if call == "enumerate":
        q, = qs
        r = ctx.run(q, mode=gem.MODE_ENUMERATE, emb_cap=state["room"])
        # embeddings come in no fixed order: one 64-bit key per embedding, sorted
        key = np.zeros(state["room"], np.uint64)
        found = key[:len(r["embeddings"])]
        for u in range(q.nv):
            found *= np.uint64(1 << (64 // q.nv))
            found += r["embeddings"][:, u]
        found.sort()
        return {"embeddings": key, "count": np.array([r["count"], r["n_written"], r["emb_hash"]], np.uint64)}
    if call == "relaxed":
        q, = qs
        out = np.zeros((1 + q.nv * (q.nv - 1) // 2, 3), np.uint64)  # room for every query of this many vertices
        for i, (mask, r) in enumerate(ctx.relaxed(q, state["threshold"])):
            out[i] = mask, r["count"], r["status_code"]
        return {"masks, counts, status": out}
    if call == "filter":
        q, = qs
        lists = ctx.filter(q, threshold=state["threshold"])
        ends = np.cumsum([len(c) for c in lists])
        out = np.zeros(state["room"], np.uint32)
        np.concatenate(lists, out=out[:ends[-1]])
        return {"ends": ends, "candidates": out}
    if call == "serve":
        return _serve(ctx, qs)
    raise ValueError(call)


def work(case):
    """Bytes that the path cannot do without: the per-vertex arrays once per call, the arcs of the vertices that can
    key a table once per call, and each edge table's expected values once (queries take labels as they occur).  A
    call of `run` or `filter` is one query's; the others share one call.  There is no floating-point work."""
    n, zipf, L = case["vertices"], case["zipf"], case["labels"]
    p = np.arange(1, L + 1, dtype=np.float64) ** -zipf
    p /= p.sum()
    same = float((p * p).sum())  # probability that a vertex has the label of a query vertex
    arcs = 2.0 * case["edge_factor"] * n * 0.9
    sizes = [s for s in MIX if s <= case.get("largest", 32)] if case["k"] == 0 else [case["k"]]
    k, q = sum(sizes) / len(sizes), case["queries"]
    calls = q if case["call"] in ("run", "enumerate", "relaxed", "filter") else 1
    rows = q / calls * k
    stride = -(-L // 16) * 16 if L <= 64 else 0
    per_call = n * (8.0 + stride)
    if case["call"] == "filter":
        return {"bytes": calls * (per_call + 4 * k * n * same), "flops": 0}
    held = 1 - (1 - same) ** rows  # share of vertices that some query vertex can map to
    per_call += 4 * arcs * held + 4 * (q / calls) * (k - 1) * arcs * same * same
    return {"bytes": calls * per_call, "flops": 0}


def tolerance(case):
    return "exact"
