"""Kernels at the sizes where they can go wrong, bit-exact against the CPU
oracle or a closed form: filter rows on graphs of ragged size and of more
labels than the resident label counts cover, membership columns of every
width, hash buckets that overflow, pair items and pair pools of odd lengths,
scans on both sides of the one-block limit."""
import math
import threading

import numpy as np
import pytest

import gem_b200 as gem
import oracle

pytestmark = pytest.mark.gpu


def cut(g, n):
    """The subgraph that the first n vertices induce."""
    off, nbr, lab = g.arrays()
    src = np.repeat(np.arange(g.nv), np.diff(off).astype(np.int64))
    keep = (src < n) & (nbr < n)
    new = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(src[keep], minlength=n), out=new[1:])
    return gem.HostGraph.from_csr(new, nbr[keep], lab[:n])


# one row to a full group of them, one tile to several sets, few labels to more than 64 (counted per wave)
@pytest.mark.parametrize("nv", [9, 31, 33, 257, 1023, 4096 - 7])
@pytest.mark.parametrize("labels", [1, 3, 23, 64, 65, 150])
def test_filter_rows(nv, labels):
    g = cut(gem.HostGraph.rmat(12, 8, seed=91), nv).set_labels(labels, 0.0, seed=7)
    rng = np.random.default_rng(nv + labels)
    lab = g.arrays()[2]
    qs = [gem.Query([lab[0]], []), gem.Query([lab[0], labels + 5], [(0, 1)])]
    for k in (2, 5, 32):  # random trees: any labels, among them ones that few vertices or none have
        qs.append(gem.Query(rng.integers(0, labels + 1, k), [(int(rng.integers(0, i)), i) for i in range(1, k)]))
    # a hub with eleven distinct neighbour labels: more needs than a row holds
    qs.append(gem.Query([0] + [i % (labels + 1) for i in range(11)], [(0, i) for i in range(1, 12)]))
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        for q in qs:
            for t in (0, 1, 2):
                got, exp = c.filter(q, threshold=t), oracle.filter(g, q, threshold=t)
                for u in range(q.nv):
                    assert np.array_equal(got[u], exp[u]), (q.nv, t, u)


# column widths: 1 word (one for all rows, then per label), 2, and multiples of 4; above 64 labels too
@pytest.mark.parametrize("labels,n,k", [(3, 2, 4), (90, 40, 6), (40, 60, 6), (16, 120, 6), (5, 120, 6), (2, 60, 5)])
def test_batch_columns(labels, n, k):
    g = cut(gem.HostGraph.rmat(10, 6, seed=17), 1001).set_labels(labels, 0.0, seed=5)
    qs = gem.gen_queries(g, k, gem.SPARSE, n, seed=labels)
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        rs = c.batch(qs)[1]
        rh = c.batch(qs, mode=gem.MODE_HASH)[1] if labels > 10 else None
        # every query alone: waves of few rows, whose table passes are another kernel
        assert [(r["status"], r["count"]) for r in rs] == [("OK", c.run(q)["count"]) for q in qs]
        if rh is not None:
            alone = [c.run(q, mode=gem.MODE_HASH) for q in qs]
            assert [(r["count"], r["emb_hash"]) for r in rh] == [(r["count"], r["emb_hash"]) for r in alone]
        for q, r in list(zip(qs, rs))[:2]:
            cand = oracle.filter(g, q)
            for a, b in q.edges.tolist():
                for u, w in ((a, b), (b, a)):
                    off, vals = c.edge_table(q, u, w)
                    eo, ev = oracle.edge_table(g, cand[u], cand[w])
                    assert np.array_equal(off, eo) and np.array_equal(vals, ev), (u, w)
    checked = 0
    for i, q in enumerate(qs):
        cnt, h, ok = oracle.count(g, q, want_hash=rh is not None, work_cap=20_000_000)
        if ok:
            checked += 1
            assert rs[i]["status"] == "OK" and rs[i]["count"] == cnt, i
            if rh is not None:
                assert rh[i]["count"] == cnt and rh[i]["emb_hash"] == h, i
    assert checked >= n // 3


# complete graphs: every neighbourhood hash holds n - 1 keys (one bucket upwards; overflows at every size), every
# intersection is long, and the counts are falling factorials
@pytest.mark.parametrize("n", [2, 3, 4, 5, 9, 33, 70])
def test_complete_graph_paths_and_cycles(n):
    g = gem.HostGraph.from_edges(n, [(i, j) for i in range(n) for j in range(i + 1, n)], [0] * n)
    shapes = [[(i, i + 1) for i in range(k - 1)] for k in (2, 3, 4, 5)]
    shapes += [s + [(0, k - 1)] for s, k in zip(shapes[1:], (3, 4, 5))]
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        for e in shapes:
            k = max(max(x) for x in e) + 1
            q, exp = gem.Query([0] * k, e), math.perm(n, k)
            assert c.run(q)["count"] == exp, (n, e)
            if exp <= 20_000_000:
                r = c.run(q, mode=gem.MODE_HASH)
                assert r["status"] == "OK" and r["count"] == exp, (n, e)


# a hub with d leaves, each with its own pendant: pair items and pools of d entries around the sizes of a warp's chunk
@pytest.mark.parametrize("d", [1, 31, 32, 33, 64, 1000, 5000])
def test_hub_and_spokes(d):
    e = [(0, 1 + i) for i in range(d)] + [(1 + i, 1 + d + i) for i in range(d)]
    g = gem.HostGraph.from_edges(1 + 2 * d, e, [0] + [1] * d + [2] * d)
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        path5 = gem.Query([2, 1, 0, 1, 2], [(0, 1), (1, 2), (2, 3), (3, 4)])
        star = gem.Query([0, 1, 1], [(0, 1), (0, 2)])
        for q, exp in ((path5, d * (d - 1)), (star, d * (d - 1)), (gem.Query([0, 1, 2], [(0, 1), (1, 2)]), d)):
            assert c.run(q)["count"] == exp
            if exp < 3_000_000:
                r = c.run(q, mode=gem.MODE_ENUMERATE, emb_cap=exp + 1)
                assert r["count"] == r["n_written"] == exp
                assert len(np.unique(r["embeddings"], axis=0)) == exp


# the one-block scan's limit is 16,384 items: candidate sets, keys, vertex and table tiles on both sides of it
@pytest.mark.parametrize("nv", [16383, 16384, 16385, 40000])
def test_scan_limit(nv):
    # a cycle: every vertex a candidate, one tile and two values per key
    g = gem.HostGraph.from_edges(nv, [(i, (i + 1) % nv) for i in range(nv)], [0] * nv)
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        assert c.run(gem.Query([0, 0, 0], [(0, 1), (1, 2)]))["count"] == 2 * nv
        off, vals = c.edge_table(gem.Query([0, 0], [(0, 1)]), 0, 1)
        assert np.array_equal(off, 2 * np.arange(nv + 1, dtype=np.uint64)) and len(vals) == 2 * nv


# queries with an automorphism that exchanges two enumerated levels (counted by one of the two orders, twice), next to
# ones that only look like it
@pytest.mark.parametrize("labels,edges", [
    ([0, 1, 1, 0], "01 12 23"), ([0, 1, 1, 2], "01 12 23"), ([0, 0, 0, 0], "01 12 23"), ([0, 1, 0, 1], "01 12 23 03"),
    ([0, 1, 0, 2], "01 12 23 03"), ([0, 0, 0], "01 12 02"), ([1, 0, 0, 2], "01 02 12 13 23"),
    ([0, 0, 0, 0], "01 02 03 12 13 23"), ([2, 1, 0, 1, 2], "01 12 23 34"), ([2, 1, 0, 1, 0], "01 12 23 34"),
    ([0, 1, 0, 1, 2], "01 12 23 03 24"), ([0, 1, 1, 0, 2, 2], "01 12 23 14 25"), ([0, 1, 1, 0, 2], "01 12 23 14")])
def test_symmetric_queries(labels, edges):
    g = cut(gem.HostGraph.rmat(10, 6, seed=23), 777).set_labels(3, 0.0, seed=11)
    q = gem.Query(labels, [(int(e[0]), int(e[1])) for e in edges.split()])
    exp, h, ok = oracle.count(g, q, want_hash=True, work_cap=2_000_000_000)
    assert ok and exp > 0
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        assert c.run(q)["count"] == exp
        r = c.run(q, mode=gem.MODE_HASH)
        assert (r["count"], r["emb_hash"]) == (exp, h)
        assert [r["count"] for r in c.batch([q] * 40)[1]] == [exp] * 40


def test_out_of_core_partitions_kept_or_streamed_twice():
    """With an ample budget the write pass reads the partitions that the count
    pass streamed; with a tight one both passes stream them.  Same counts."""
    g = gem.HostGraph.rmat(16, 8, seed=0x47454D10).set_labels(8, 0.0, seed=3)
    qs = gem.gen_queries(g, 4, gem.ANY, 5, seed=8)
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        exp = [c.run(q)["count"] for q in qs]
    streamed = []
    for budget in (0, 72 << 20):  # the adjacency is 3.8 MB: more than a sixteenth of what 72 MiB leaves
        with gem.Context(time_cap_ms=20000, ooc=True, ooc_stream=1, ooc_part_kib=256, budget_bytes=budget) as c:
            c.load_graph(g)
            assert [c.run(q)["count"] for q in qs] == exp
            assert [r["count"] for r in c.batch(qs[:2])[1]] == exp[:2]
            s = c.ooc_stats()
            assert s["waves_in_place"] == 0
            streamed.append(s["bytes_streamed"])
    assert streamed[1] == 2 * streamed[0]


def test_lanes_of_different_column_widths():
    """The count pass of wide columns (64 words: 2,032 filter rows of one label) takes more shared memory than a kernel
    may by default: that limit is the kernel's, so waves of another width on another thread must leave it."""
    g = gem.HostGraph.rmat(11, 6, 0.25, 0.25, 0.25, seed=29).set_labels(2100, 0.0, seed=3)
    off, nbr, lab = g.arrays()
    u = np.repeat(np.arange(g.nv), np.diff(off).astype(np.int64))[::300][:60]
    edges = [gem.Query([lab[a], lab[b]], [(0, 1)]) for a, b in zip(u, nbr[::300])]
    spine = [(i, i + 1) for i in range(15)] + [(i, 16 + i) for i in range(16)]
    chains = [gem.Query([0] * 16 + list(range(16 * i, 16 * i + 16)), spine) for i in range(127)]
    widths = [chains + edges[:8], edges]
    with gem.Context(time_cap_ms=20000) as a, gem.Context(time_cap_ms=20000) as b:
        exp, bad = [], []
        for c, qs in zip((a, b), widths):
            c.load_graph(g)
            exp.append(c.batch_counts(qs)[1].tolist())
        assert min(exp[1]) > 0 and exp[0][127:] == exp[1][:8]

        def lane(i, c):
            for _ in range(400):
                st, counts, status = c.batch_counts(widths[i])
                if st != 0 or status.any() or counts.tolist() != exp[i]:
                    bad.append((i, st))

        lanes = [threading.Thread(target=lane, args=x) for x in ((0, a), (1, b))]
        for t in lanes:
            t.start()
        for t in lanes:
            t.join()
        assert not bad, (len(bad), bad[0])


@pytest.mark.parametrize("kind", ["auto", "cuckoo"])
def test_calls_after_a_failed_one(kind):
    """Calls that run out of budget at every phase (budgets in small steps) leave copies in flight; the calls right
    after them, which use the same staging buffer, are exact."""
    g = gem.HostGraph.rmat(13, 8, seed=41).set_labels(5, 0.0, seed=2)
    opts = dict(time_cap_ms=20000, index_kind=gem.IDX_CUCKOO if kind == "cuckoo" else gem.IDX_AUTO)
    big = gem.gen_queries(g, 20, gem.ANY, 1, seed=3)[0]
    small = gem.gen_queries(g, 3, gem.ANY, 3, seed=8)
    with gem.Context(**opts) as c:
        c.load_graph(g)
        exp = [(c.run(q)["count"], [x.tolist() for x in c.filter(q)]) for q in small]
    failed = 0
    for kib in range(6 << 10, 64 << 10, 32):
        try:
            c = gem.Context(budget_bytes=kib << 10, **{**opts, "time_cap_ms": 100})
            c.load_graph(g)
        except gem.GemError:
            continue
        ran = 0
        with c:
            for q, e in zip(small, exp):
                r = c.run(big, raise_on_error=False)
                assert r["status"] in ("OK", "ERR_OOM", "ERR_TIMEOUT"), r
                ran += r["status"] != "ERR_OOM"
                failed += r["status"] == "ERR_OOM"
                try:
                    got = (c.run(q)["count"], [x.tolist() for x in c.filter(q)])
                except gem.GemError as x:
                    assert x.status == 2, x
                    continue
                assert got == e
        if ran == len(small):
            break
    assert failed > 30


@pytest.mark.parametrize("kind", ["auto", "cuckoo"])
def test_optional_memory_gives_way(kind):
    """Key positions that only spread the join's items are optional: budgets that hold everything else run the batch
    in one wave, whether the positions or what is allocated after them would not have fitted."""
    g = gem.HostGraph.rmat(14, 8, seed=51).set_labels(8, 0.0, seed=2)
    qs = gem.gen_queries(g, 4, gem.ANY, 12, seed=4)
    opts = dict(time_cap_ms=20000, index_kind=gem.IDX_CUCKOO if kind == "cuckoo" else gem.IDX_AUTO)
    with gem.Context(**opts) as c:
        c.load_graph(g)
        rs = c.batch(qs, mode=gem.MODE_HASH)[1]
        exp = [(r["count"], r["emb_hash"]) for r in rs]
        whole = c.ooc_stats()["resident_bytes"] + rs[0]["arena_bytes"]
        optional = 4 * rs[0]["table_total"]
    assert optional > 400_000
    for less in (0, 256, 4096, 65536, optional // 4, optional // 2, optional - 4096):
        with gem.Context(budget_bytes=whole - less, **opts) as c:
            c.load_graph(g)
            st, rs = c.batch(qs, mode=gem.MODE_HASH)
            assert st == 0 and len({r["wave"] for r in rs}) == 1, (less, st)
            assert [(r["count"], r["emb_hash"]) for r in rs] == exp


def test_pool_counts_survive_the_cap():
    """The depth-first part runs out of time: queries of the pools, counted whole before it, keep their counts, also
    the ones that come after its queries in the join's order."""
    g = gem.HostGraph.rmat(18, 16, seed=61).set_labels(8, 1.0, seed=2)
    # three vertices of one label next to both ends of an edge: seven subsets, too many for the pair pool
    slow = gem.Query([0] * 5, [(0, 1)] + [(e, i) for e in (0, 1) for i in (2, 3, 4)])
    fast = [gem.Query([7, 6, 6, 7], [(0, 1), (1, 2), (2, 3)]),  # two levels like it, and fewer vertices
            gem.Query([7, 7, 3, 4, 5, 6], [(0, 1), (0, 2), (0, 3), (1, 4), (1, 5)])]  # two levels, and more
    with gem.Context(time_cap_ms=60000) as c:
        c.load_graph(g)
        exp = [c.run(q)["count"] for q in fast]
    with gem.Context(time_cap_ms=3) as c:
        c.load_graph(g)
        rs = c.batch([slow] + fast)[1]
    assert rs[0]["status"] == "ERR_TIMEOUT"
    assert [(r["status"], r["count"]) for r in rs[1:]] == [("OK", e) for e in exp]


@pytest.mark.parametrize("ooc", [False, True])
def test_more_labels_than_resident_counts(ooc):
    """Above 64 labels the filter counts neighbour labels on the way: rows of one label whose neighbours have more
    labels than a group counts, lists of up to 1,500 arcs read in part or whole, batches against single runs."""
    g = cut(gem.HostGraph.rmat(13, 16, seed=71), 8000).set_labels(300, 1.0, seed=5)
    off, nbr, lab = g.arrays()
    off = off.astype(np.int64)
    rng = np.random.default_rng(9)
    centres = np.flatnonzero((lab == 0) & (np.diff(off) > 8))
    assert np.diff(off)[centres].max() > 1000
    stars = []
    for v in rng.choice(centres, 150):
        leaf = lab[rng.choice(nbr[off[v]:off[v + 1]], rng.integers(2, 6), replace=False)]
        stars.append(gem.Query([0] + leaf.tolist(), [(0, 1 + i) for i in range(len(leaf))]))
    hub = centres[np.argmax(np.diff(off)[centres])]
    wide = gem.Query([0] + lab[rng.choice(nbr[off[hub]:off[hub + 1]], 31, replace=False)].tolist(),
                     [(0, 1 + i) for i in range(31)])
    with gem.Context(time_cap_ms=20000, ooc=ooc) as c:
        c.load_graph(g)
        for q in stars[:4] + [wide, gem.Query([0, 299, 0, 301], [(0, 1), (1, 2), (2, 3)])]:
            for t in (0, 1, 3):
                for a, b in zip(c.filter(q, threshold=t), oracle.filter(g, q, threshold=t)):
                    assert np.array_equal(a, b), t
        st, counts, status = c.batch_counts(stars)
        assert st == 0 and len({tuple(q.labels) for q in stars}) > 100
        assert counts.tolist() == [c.run(q)["count"] for q in stars]
        for q, n in list(zip(stars, counts))[:20]:
            exp, _, ok = oracle.count(g, q, want_hash=False, work_cap=20_000_000)
            assert not ok or exp == n


def test_many_labels_take_no_memory():
    """A batch on a graph of many labels runs in one wave on the bytes that it holds at its end."""
    g = gem.HostGraph.rmat(18, 4, 0.25, 0.25, 0.25, seed=73).set_labels(300, 0.0, seed=5)
    qs = gem.gen_queries(g, 5, gem.ANY, 60, seed=6)
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        rs = c.batch(qs)[1]
        exp = [r["count"] for r in rs]
        whole = c.ooc_stats()["resident_bytes"] + rs[0]["arena_bytes"]
    with gem.Context(time_cap_ms=20000, budget_bytes=whole) as c:
        c.load_graph(g)
        st, rs = c.batch(qs)
        assert st == 0 and len({r["wave"] for r in rs}) == 1
        assert [r["count"] for r in rs] == exp


# waves of one column word for all rows, and of one per label
@pytest.mark.parametrize("n", [1, 30])
def test_filter_bytes(n):
    """The filter's algorithmic bytes: labels, label counts of the rows' labels (16 a vertex), three passes of words,
    candidate lists."""
    g = gem.HostGraph.rmat(10, 6, seed=81).set_labels(7, 0.0, seed=5)
    qs = gem.gen_queries(g, 5, gem.ANY, n, seed=6)

    def row(q, u):
        return q.labels[u], tuple(sorted(q.labels[a + b - u] for a, b in q.edges.astype(int).tolist() if u in (a, b)))

    sigs = {row(q, u) for q in qs for u in range(q.nv)}
    assert (len(sigs) <= 32) == (n == 1)
    freq = np.bincount(g.arrays()[2], minlength=7)
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        cand = {}
        for q in qs:
            for u, x in enumerate(c.filter(q)):
                cand[row(q, u)] = len(x)
        got = c.batch(qs)[1][0]["bytes_alg"][0]
    words = g.nv // 32
    assert got == (4 * g.nv + 16 * sum(int(freq[x]) for x in {s[0] for s in sigs}) + 16 * words * len(sigs)
                   + 4 * sum(cand.values()))


# hubs (units of four tiles where columns are narrow) and equal degrees; targets in one, two and more words of columns
# that are up to 24 words wide for the rows that key tables
@pytest.mark.parametrize("skew", [True, False])
@pytest.mark.parametrize("leaf,n", [(6, 60), (6, 240), (12, 700)])
def test_sources_wider_than_targets(skew, leaf, n):
    p = (0.57, 0.19, 0.19) if skew else (0.25, 0.25, 0.25)
    g = gem.HostGraph.rmat(12, 12, *p, seed=91).set_labels(14, 0.5, seed=4)
    rng = np.random.default_rng(n)
    qs = [gem.Query([0] + np.sort(rng.integers(1, 1 + leaf, 4)).tolist(), [(0, i) for i in range(1, 5)]) for _ in range(n)]
    # leaves with leaves of their own: rows of label 1 that tables target, some of them beyond the first words
    qs += [gem.Query([0, 1, a, b], [(0, 1), (1, 2), (1, 3)]) for a in range(1, leaf) for b in range(a + 1)][:n // 4]
    with gem.Context(time_cap_ms=20000) as c:
        c.load_graph(g)
        st, counts, status = c.batch_counts(qs)
        assert st == 0 and int(counts.sum()) > 0
        assert counts.tolist() == [c.run(q)["count"] for q in qs]
