"""GPU tests of the tables an engine keeps: their size follows the graph's, the pair table starts over when its
phase numbers run out, kept sets longer than one piece, and the seed tables of many plans."""
import ctypes

import numpy as np
import pytest

import csm
from csm import DataGraph, QueryGraph
from helpers import cycle, random_graph
from oracle import Oracle

pytestmark = pytest.mark.gpu


def query(labels, edges):
    s, d = zip(*edges)
    return QueryGraph(np.array(labels, dtype=np.uint32), np.array(s, dtype=np.uint32), np.array(d, dtype=np.uint32),
                      np.zeros(len(edges), dtype=np.uint32))


def free_bytes(eng):
    free, total = ctypes.c_uint64(), ctypes.c_uint64()
    assert eng.lib.csm_device_memory(eng._h, ctypes.byref(free), ctypes.byref(total)) == 0
    return free.value


def test_small_engines_stay_small():
    """A 4-cycle's tail is a pair intersection: the pair table of an engine over 30,000 edges must not take the
    64 MB that a large graph's takes."""
    rng = np.random.default_rng(5)
    vl, s, d, el = random_graph(6000, 30000, 2, rng)
    engines = [csm.Engine(max_batch=64, frontier_bytes=1 << 20, queue_slots=1024) for _ in range(5)]
    for e in engines:
        e.load_query(cycle(4, [0, 1, 0, 1]))
    engines[0].load_graph(DataGraph(vl, s, d, el))  # takes what the device needs for the kernels, too
    before = free_bytes(engines[0])
    for e in engines[1:]:
        e.load_graph(DataGraph(vl, s, d, el))
    each = (before - free_bytes(engines[0])) / 4
    for e in engines:
        e.close()
    assert each < 32 << 20, f"{each / 2 ** 20:.0f} MB an engine"


def test_tables_grow_with_the_pool():
    """From a nearly empty graph and pool to one that needs larger ones: counts equal the oracle's all the way."""
    rng = np.random.default_rng(6)
    vl, s, d, el = random_graph(3000, 40000, 2, rng)
    q = cycle(4, [0, 1, 0, 1])
    start = 1000
    data = DataGraph(vl, s[:start], d[:start], el[:start])
    eng = csm.Engine(max_batch=64, pool_entries=1 << 14)
    eng.load_query(q)
    eng.load_graph(data)
    oracle = Oracle(q, data)
    small = eng.stats().pool_capacity
    total = 0
    for at in range(start, len(s), 6500):
        b = csm.Batch(s[at:at + 6500], d[at:at + 6500], el[at:at + 6500])
        for x in (b, csm.Batch(b.src, b.dst, b.elabels, (rng.random(len(b.src)) < 0.3).astype(np.uint8))):
            res, r = eng.apply(x)[0], oracle.apply(x)
            assert (res.positive, res.negative) == (r["pos"], r["neg"])
            total += r["pos"] + r["neg"]
    st = eng.stats()
    eng.close()
    assert total > 0 and st.compactions > 0 and st.pool_capacity > 64 * small // 8


@pytest.mark.parametrize("config", [dict(), dict(search_strategy=0, cuda_graphs=1)])
def test_pair_table_starts_over(config):
    """The table's entries carry a phase number that starts over after the first 16 batches: sizes kept under the
    same number before that must not be taken for this phase's."""
    rng = np.random.default_rng(8)
    vl, s, d, el = random_graph(300, 6000, 2, rng)
    q = cycle(4, [0, 1, 0, 1])
    keep = 3000
    data = DataGraph(vl, s[:keep], d[:keep], el[:keep])
    eng = csm.Engine(max_batch=300, **config)
    eng.load_query(q)
    eng.load_graph(data)
    oracle = Oracle(q, data)
    for i in range(40):
        pick = rng.integers(0, len(s), size=300)
        b = csm.Batch(s[pick], d[pick], el[pick], (rng.random(300) < 0.5).astype(np.uint8))
        res, r = eng.apply(b)[0], oracle.apply(b)
        assert (res.positive, res.negative) == (r["pos"], r["neg"]), f"batch {i}"
        assert r["pos"] > 0 and r["neg"] > 0
    eng.close()


def test_sets_longer_than_one_piece():
    """A tail vertex with three lists, two of them of prefix hubs that share 224, 225, 257 or 700 neighbours: the
    kept intersection is made in pieces of at most 256.  Other query vertices of the tail's label sit in it."""
    k4 = [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (2, 3)]
    queries = [query([0, 1, 2, 3], k4), query([0, 1, 2, 3, 0], k4 + [(0, 4)]), query([0, 1, 2, 3, 3], k4 + [(0, 4), (1, 4)]),
               query([0, 1, 3, 3, 0], k4 + [(0, 4)])]
    rng = np.random.default_rng(9)
    shared = [224, 225, 257, 700]
    a, b, c = np.arange(4), np.arange(4, 8), np.arange(8, 48)   # hubs of labels 0 and 1, vertices of label 2
    t = np.arange(48, 48 + 900)                                  # label 3
    x = np.arange(948, 988)                                      # leaves of label 0
    vl = np.zeros(988, dtype=np.uint32)
    vl[b], vl[c], vl[t] = 1, 2, 3
    edges = set()
    for i, k in enumerate(shared):  # hub i of label 0 and hub i of label 1 share exactly t[0..k-1]
        edges |= {(int(a[i]), int(v)) for v in t[:k]} | {(int(b[i]), int(v)) for v in t[:k]}
        edges |= {(int(a[i]), int(b[i]))} | {(int(h), int(w)) for h in (a[i], b[i]) for w in c[rng.random(40) < 0.5]}
        edges |= {(int(a[i]), int(v)) for v in x[10 * i:10 * i + 10]}
    edges |= {(int(w), int(v)) for w in c for v in t[rng.random(900) < 0.2]}
    edges |= {(int(t[i]), int(t[j])) for i, j in zip(rng.integers(0, 300, 3000), rng.integers(300, 900, 3000))}
    e = np.array(sorted(edges), dtype=np.uint32)
    hubs = (e[:, 0] < 4) & (e[:, 1] < 8)  # the hubs' own edges open the widest prefixes
    part = rng.random(len(e)) < 0.04
    part |= hubs
    data = DataGraph(vl, e[~part, 0], e[~part, 1], np.zeros((~part).sum(), dtype=np.uint32))
    with csm.Engine() as eng:
        for q in queries:
            eng.load_query(q)
        eng.load_graph(data)
        oracles = [Oracle(q, data) for q in queries]
        n = int(part.sum())
        for dele in (np.zeros(n, np.uint8), (rng.random(n) < 0.5).astype(np.uint8), np.ones(n, np.uint8)):
            batch = csm.Batch(e[part, 0], e[part, 1], np.zeros(n, dtype=np.uint32), dele)
            res = eng.apply(batch)
            for qi, o in enumerate(oracles):
                r = o.apply(batch)
                assert (res[qi].positive, res[qi].negative) == (r["pos"], r["neg"]), f"query {qi}"
                assert r["pos"] + r["neg"] > 0


def test_more_plans_than_one_block_finds_ranges_for():
    """Over 128 query edges the seed ranges and the ticket prefix come from two launches instead of one."""
    rng = np.random.default_rng(12)
    vl, s, d, el = random_graph(500, 5000, 3, rng)
    queries = [cycle(4, rng.integers(0, 3, size=4)) for _ in range(30)] + [cycle(3, rng.integers(0, 3, size=3)) for _ in range(8)]
    assert sum(len(q.src) for q in queries) > 128
    keep = 4200
    data = DataGraph(vl, s[:keep], d[:keep], el[:keep])
    with csm.Engine() as eng:
        for q in queries:
            eng.load_query(q)
        eng.load_graph(data)
        oracles = [Oracle(q, data) for q in queries]
        seen = 0
        for pick in np.array_split(rng.permutation(len(s))[:1500], 3):
            b = csm.Batch(s[pick], d[pick], el[pick], (pick < keep).astype(np.uint8))
            res = eng.apply(b)
            for qi, o in enumerate(oracles):
                r = o.apply(b)
                assert (res[qi].positive, res[qi].negative) == (r["pos"], r["neg"]), f"query {qi}"
                assert eng.edge_counts(qi) == (r["per_qe_pos"], r["per_qe_neg"]), f"query {qi} per-edge split"
                seen += r["pos"] > 0 and r["neg"] > 0
        assert seen > len(queries)
