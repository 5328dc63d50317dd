"""Representative calls of the engine's public entry points, for timing.

A case is a standing query set over a data graph of one of the benchmark configurations
(csm.gen.CONFIGS) and one update batch.  A pass applies the batch and then its inverse, which puts
the graph back, so passes can repeat: the first half counts what the batch creates and destroys, the
second half runs the same updates the other way round (insertions become deletions).  Graphs and
batches are drawn from the seed; the queries are the configurations' own, written out below, because
a standing query is part of what a user's program is, not of its data.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gcsm-bu_b200"))
import csm  # noqa: E402

# Shapes of the data graphs (Chung-Lu exponent, label counts and skews as in csm.gen.CONFIGS) and
# the range of batch sizes their use calls for.
GRAPHS = {
    # Plain method (c1): a small graph kept by a latency-bound caller.
    "plain": dict(n=10_000, m=50_000, gamma=2.3, nvl=4, vzipf=0.0, nel=1, ezipf=0.0, cap=False, lo=64, hi=4096),
    # Amazon-shaped (c2, c4): Zipf(1.0) labels, 65,536-update batches.
    "amazon": dict(n=400_000, m=2_400_000, gamma=2.1, nvl=6, vzipf=1.0, nel=1, ezipf=0.0, cap=True, lo=256, hi=65_536),
    # Netflow-shaped (c5): edge labels, batches of 1k to 256k.
    "netflow": dict(n=3_000_000, m=20_000_000, gamma=2.1, nvl=8, vzipf=0.0, nel=16, ezipf=1.1, cap=True, lo=1_024,
                    hi=262_144),
    # LiveJournal-shaped (c3): heavy vertices, 1M-update batches.
    "livejournal": dict(n=4_800_000, m=43_000_000, gamma=1.9, nvl=20, vzipf=1.2, nel=1, ezipf=0.0, cap=True, lo=65_536,
                        hi=1_000_000),
}

# Standing queries: vertex labels, then edges a-b or a-b:label.
QUERIES = {
    "plain": ["1,3,1,3 0-1,1-2,2-3,3-0"],
    "amazon": [
        "0,0,1,1,2,5 0-1,0-5,1-2,1-3,1-4,2-3,2-4,2-5,4-5",
        "4,0,1,2,3,0 0-1,0-2,0-3,0-4,0-5,1-2,2-3,2-5,3-4",
        "0,0,0,5,2,0 0-1,1-2,1-3,1-4,2-3,2-4,2-5,3-4,4-5",
        "0,0,3,0,0,1 0-1,1-2,1-4,1-5,2-3,2-4,2-5,3-4,4-5",
        "3,0,1,4,0,0 0-1,0-2,0-3,0-4,1-2,1-4,1-5,2-3,2-4,4-5",
        "2,2,0,1,0,5 0-1,1-2,2-3,3-4,4-5",
        "4,4,0,1,4,0 0-1,0-2,2-3,3-4,4-5",
    ],
    "netflow": [
        "5,5,6,1,7,7,7 0-1:9,1-2:0,1-3:4,1-4:1,1-5:4,1-6:1,3-4:5,3-5:0,3-6:0,4-5:0,5-6:2",
        "3,4,6,3,1,5,7 0-1:5,1-2:5,2-3:6,3-4:0,4-5:0,5-6:3,1-6:1",
        "7,3,0,5 0-1:6,1-2:11,1-3:2,2-3:7",
        "7,7,0,6,0,6 0-1:7,1-2:0,2-3:3,3-4:0,4-5:1,1-4:0",
        "4,3,6,7,4,1 0-1:0,1-2:14,1-4:4,1-5:0,2-3:2,2-4:0,2-5:0,3-4:0,4-5:6",
        "5,4,0,4,7 0-1:6,0-2:0,0-3:8,1-4:3,2-3:3,2-4:0,3-4:0",
        "3,7,3,1,3,1,5,0 0-1:0,1-2:11,2-3:1,3-4:0,4-5:0,5-6:1,6-7:8,1-6:1,3-6:0,1-5:0",
        "3,6,6,5,2,5,1 0-1:1,1-2:0,1-5:0,1-6:0,2-3:1,2-4:0,2-6:3,3-4:0,3-5:7,3-6:0,4-6:2,5-6:7",
    ],
    "livejournal": [
        "14,11,14,8,15,16,11,16 0-1,0-4,1-2,1-3,1-4,1-5,2-7,4-5,4-6,4-7,5-7,6-7",
        "12,19,13,14,19,16,19,10 0-1,0-2,1-2,1-4,1-6,2-3,2-4,2-5,2-6,2-7,3-4,3-5,3-7,4-5,4-6",
        "17,17,16,14,12,18,12,8 0-1,1-2,2-3,2-4,2-5,2-6,3-4,3-5,3-7,4-5,4-6,4-7",
        "11,13,8,11,13,14,18,17 0-1,1-2,1-3,1-5,1-6,2-3,3-4,3-5,3-6,4-7,5-7,6-7",
    ],
}


def parse_query(text):
    labels, edges = text.split()
    pairs = [e.split(":") for e in edges.split(",")]
    ends = [tuple(map(int, p[0].split("-"))) for p in pairs]
    return csm.QueryGraph(np.array(labels.split(","), dtype=np.uint32), np.array([a for a, _ in ends], dtype=np.uint32),
                          np.array([b for _, b in ends], dtype=np.uint32),
                          np.array([int(p[1]) if len(p) > 1 else 0 for p in pairs], dtype=np.uint32))


def zipf(k, s):
    p = np.arange(1, k + 1, dtype=np.float64) ** -s
    return p / p.sum()


def shape(case):
    """The case's graph: its configuration with vertices and edges scaled, and the weights of its vertices."""
    g = dict(GRAPHS[case["graph"]])
    g["n"], g["m"] = max(64, int(g["n"] * case["scale"])), max(256, int(g["m"] * case["scale"]))
    w = (np.arange(g["n"], dtype=np.float64) + 1.0) ** (-1.0 / (g["gamma"] - 1.0))
    w *= 2.0 * g["m"] / w.sum()
    return g, np.minimum(w, math.sqrt(w.sum())) if g["cap"] else w


def inputs(case, seed):
    """Vertex labels, the initial edges (src, dst, label) and the batch (src, dst, label, delete), on the GPU."""
    g, w = shape(case)
    n, m = g["n"], g["m"]
    gen = torch.Generator("cuda").manual_seed(seed)
    cdf = torch.from_numpy(np.cumsum(w / w.sum())).cuda()

    def draw(count, c):
        return torch.searchsorted(c, torch.rand(count, generator=gen, device="cuda", dtype=torch.float64)).clamp_(max=len(c) - 1)

    def labels(count, k, s):
        return draw(count, torch.from_numpy(np.cumsum(zipf(k, s))).cuda())

    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    while len(keys) < m:
        more = int((m - len(keys)) * 1.3) + 1024
        a, b = draw(more, cdf), draw(more, cdf)
        keys = torch.unique(torch.cat([keys, (torch.minimum(a, b) * n + torch.maximum(a, b))[a != b]]))
    keys = keys[torch.randperm(len(keys), generator=gen, device="cuda")[:m]]
    place = torch.randperm(n, generator=gen, device="cuda")  # hubs are not clustered at small ids
    a, b = place[keys // n], place[keys % n]
    swap = torch.rand(m, generator=gen, device="cuda") < 0.5
    a, b = torch.where(swap, b, a), torch.where(swap, a, b)
    vl, el = labels(n, g["nvl"], g["vzipf"]), labels(m, g["nel"], g["ezipf"])
    # A tenth of the edges are held out; the batch inserts some of them and deletes initial ones.
    dels = int(round(case["updates"] * case["deletes"]))
    held = max(m // 10, case["updates"] - dels)
    pick = torch.cat([torch.arange(case["updates"] - dels, device="cuda"), held + torch.arange(dels, device="cuda")])
    pick = pick[torch.randperm(len(pick), generator=gen, device="cuda")]
    return (vl.int(), (a[held:].int(), b[held:].int(), el[held:].int()),
            (a[pick].int(), b[pick].int(), el[pick].int(), (pick >= held).to(torch.uint8)))


def queries_of(case):
    return [parse_query(QUERIES[case["graph"]][int(i)]) for i in str(case["queries"]).split(",")]


def load(case, data, queries):
    eng = csm.Engine(device=0, max_batch=case["updates"], algorithm=case["algorithm"], cuda_graphs=int(case["graphs"]),
                     materialize_rows=case["rows"])
    for q in queries:
        eng.load_query(q)
    eng.load_graph(data)
    return eng


def prepare(case, seed):
    vl, graph, (s, d, l, dele) = inputs(case, seed)
    host = [x.cpu().numpy().view(np.uint32) for x in (vl, *graph)]
    data, queries = csm.DataGraph(*host), queries_of(case)
    mixed = 0.0 < case["deletes"] < 1.0
    state = {"entry": case["entry"], "rows": case["rows"], "n": case["updates"]}
    if case["entry"] == "served":
        # One tenant per standing query, all on their own copy of the graph.
        state["engines"] = [load(case, data, [q]) for q in queries]
        state["server"] = csm.Server(device=0, slots=4)
        for e in state["engines"]:
            state["server"].add_tenant(e)
    else:
        state["engine"] = load(case, data, queries)
    if case["entry"] in ("host", "served"):
        # Update arrays as a program that streams them keeps them: in pinned memory.
        arrays = [x.cpu().pin_memory() for x in (s, d, l, dele, 1 - dele)]
        state["pinned"] = arrays
        s, d, l, dele, back = [x.numpy() if x.dtype == torch.uint8 else x.numpy().view(np.uint32) for x in arrays]
        state["batches"] = [csm.Batch(s, d, l, dele if mixed or case["deletes"] else None),
                            csm.Batch(s, d, l, back if mixed or not case["deletes"] else None)]
    else:
        state["arrays"] = [(s, d, l, dele), (s, d, l, 1 - dele)]
    return state


def read(eng, results, rows):
    """What a caller reads after a batch: per query the counts, and their split by query edge or the rows."""
    out = []
    for q, r in enumerate(results):
        out.append(np.array([r.positive, r.negative, r.inserted, r.deleted], dtype=np.int64))
        if rows:
            for sign in (1, -1):  # in an array of the size the caller keeps for them
                got = eng.embeddings(q, sign).view(np.int32)
                out.append(np.full((rows, got.shape[1]), -1, dtype=np.int32))
                out[-1][:len(got)] = got
        elif len(results) <= 4:
            out.append(np.array(eng.edge_counts(q), dtype=np.int64))
    return out


def run(state):
    out, eng = [], state.get("engine")
    if state["entry"] == "served":
        ids = [state["server"].submit(b) for b in state["batches"]]
        for i in ids:
            for r in state["server"].wait(i)[1]:
                out.append(np.array([r.positive, r.negative, r.inserted, r.deleted], dtype=np.int64))
    elif state["entry"] == "host":
        for b in state["batches"]:
            out += read(eng, eng.apply(b), state["rows"])
    else:
        call = eng.apply_device if state["entry"] == "device" else eng.apply_device_static
        stream = torch.cuda.current_stream().cuda_stream
        for s, d, l, dele in state["arrays"]:
            r = call(state["n"], s.data_ptr(), d.data_ptr(), l.data_ptr(), dele.data_ptr(), stream)
            out += read(eng, r, state["rows"])
    return out


def work(case):
    """Both batches read (13 bytes an update), and for each update that matches a relation of the queries
    its two adjacency lists read and written once per batch, no list more often than that."""
    g, w = shape(case)
    pv, pe = zipf(g["nvl"], g["vzipf"]), zipf(g["nel"], g["ezipf"])
    rel = set()
    for q in queries_of(case):
        for a, b, l in zip(q.src, q.dst, q.elabels):
            rel |= {(int(q.vlabels[a]), int(l), int(q.vlabels[b])), (int(q.vlabels[b]), int(l), int(q.vlabels[a]))}
    share = sum(pv[a] * pe[l] * pv[b] for a, l, b in rel)  # of the directed edges
    # The list of an edge's end, restricted to one relation: size-biased degree, a label's part of it.
    length = 1.0 + float((w * w).sum() / w.sum()) * share / max(1, len(rel)) ** 0.5
    lists = min(case["updates"] * 2 * share * length, 2.0 * g["m"] * share)
    tenants = len(queries_of(case)) if case["entry"] == "served" else 1
    return {"bytes": 2.0 * tenants * (13 * case["updates"] + 8 * lists) + 32 * len(queries_of(case)), "flops": 0}


def tolerance(case):
    return "exact"  # counts and vertex ids


def exact(case, seed):
    """Positive and negative counts of a small case, from plain joins over the whole graph before and after."""
    if case["graph"] != "plain" or case["rows"] or case["entry"] == "served":
        return None
    vl, (s, d, l), (us, ud, ul, dele) = inputs(case, seed)
    n, q = len(vl), queries_of(case)[0]
    vl = vl.long()

    def keys(a, b):
        return torch.cat([a.long() * n + b.long(), b.long() * n + a.long()])

    gone = dele.bool()
    kept = torch.sort(keys(s, d))[0]
    kept = kept[~torch.isin(kept, keys(us[gone], ud[gone]))]  # the graph without the deleted edges
    before = torch.sort(torch.cat([kept, keys(us[gone], ud[gone])]))[0]
    after = torch.sort(torch.cat([kept, keys(us[~gone], ud[~gone])]))[0]
    nb = [[] for _ in range(q.nv)]
    for a, b in zip(q.src.tolist(), q.dst.tolist()):
        nb[max(a, b)].append(min(a, b))  # the written-out queries list every vertex after one of its neighbours

    def count(graph):
        first = torch.searchsorted(graph, torch.arange(n + 1, device="cuda") * n)
        rows = torch.nonzero(vl == int(q.vlabels[0]))
        for u in range(1, q.nv):
            at = rows[:, nb[u][0]]
            size = first[at + 1] - first[at]
            back = torch.repeat_interleave(torch.arange(len(rows), device="cuda"), size)
            step = torch.arange(len(back), device="cuda") - torch.repeat_interleave(torch.cumsum(size, 0) - size, size)
            v = graph[first[at][back] + step] % n
            ok = vl[v] == int(q.vlabels[u])
            rows, v = rows[back[ok]], v[ok]
            ok = (rows != v[:, None]).all(1)
            for p in nb[u][1:]:
                k = rows[:, p] * n + v
                ok &= graph[torch.searchsorted(graph, k).clamp_(max=len(graph) - 1)] == k
            rows = torch.cat([rows[ok], v[ok, None]], 1)
        return len(rows)

    base, pos = count(kept), count(after)
    neg, pos = count(before) - base, pos - base
    return [np.array([pos, neg], dtype=np.float64), None, np.array([neg, pos], dtype=np.float64), None]


def case(name, graph, queries, updates, deletes, entry="host", scale=1.0, algorithm=0, graphs=False, rows=0):
    return {"name": name, "graph": graph, "queries": queries, "updates": updates, "deletes": deletes, "entry": entry,
            "scale": scale, "algorithm": algorithm, "graphs": graphs, "rows": rows}


def listed():
    return [
        # A watcher that applies each small burst of new edges as it comes: latency and launches count.
        case("plain_cycle4_64", "plain", "0", 64, 0.0),
        # The plain configuration's own batch, replayed from a captured graph by a latency-bound caller
        # with the QO-GAMMA preset (depth first with work stealing).
        case("plain_cycle4_1024_graph", "plain", "0", 1024, 0.0, algorithm=2, graphs=True),
        # A caller that wants the embeddings themselves and not their number.
        case("plain_rows_4001", "plain", "0", 4001, 0.3, rows=1 << 16),
        # A small batch on a resident medium graph, in a process that may not allocate device memory.
        case("amazon_dense6_257_static", "amazon", "0", 257, 0.1, entry="static"),
        # The Amazon-shaped configuration's batch, a dense and a tree query.
        case("amazon_dense6_65536", "amazon", "2", 65_536, 0.1),
        case("amazon_tree6_65536", "amazon", "5", 65_536, 0.1),
        # Several standing queries over one graph in one engine, at a batch size of no round number.
        case("amazon_mixed4_16411", "amazon", "0,1,5,6", 16_411, 0.1),
        # Edge-labelled stream: the largest batch of its range for one selective query, and a small batch
        # for eight standing queries.
        case("netflow_sparse7_262144", "netflow", "1", 262_144, 0.3, entry="device"),
        case("netflow_mixed8_4099", "netflow", "0,1,2,3,4,5,6,7", 4_099, 0.3),
        # The serving loop: four tenants, a request and its inverse in flight.
        case("netflow_served4_8192", "netflow", "1,3,4,6", 8_192, 0.3, entry="served", scale=0.1),
        # Heavy vertices: an insertion-only stream from host memory, and the largest batch, half deletions.
        case("livejournal_dense8_250007", "livejournal", "2", 250_007, 0.0),
        case("livejournal_dense8_1000000", "livejournal", "3", 1_000_000, 0.5, entry="device"),
    ]


def draw(rng):
    graph = rng.choice(["plain", "amazon", "amazon", "netflow", "netflow", "livejournal"])
    g, pool = GRAPHS[graph], len(QUERIES[graph])
    scale = 1.0 if graph == "plain" else round(math.exp(rng.uniform(math.log(0.1), 0.0)), 3)
    hi = min(g["hi"], int(0.08 * g["m"] * scale))
    updates = int(math.exp(rng.uniform(math.log(min(g["lo"], hi // 4)), math.log(hi))))
    deletes = rng.choice([0.0, 0.1, 0.3, 0.5, 1.0])
    entry = rng.choice(["host", "host", "device", "static"] + (["served"] if graph in ("amazon", "netflow") else []))
    count = 1 if graph in ("plain", "livejournal") else rng.choice([1, 1, 2, 3, 4])
    if entry == "served":
        count, scale, updates = max(2, count), min(scale, 0.2), min(updates, int(0.02 * g["m"] * min(scale, 0.2)))
    queries = ",".join(str(i) for i in sorted(rng.sample(range(pool), count)))
    extra = rng.choice([{}, {"algorithm": 2, "graphs": True}, {"rows": 1 << 16}]) if graph == "plain" else {}
    if extra.get("rows"):
        entry = "host"
    c = case("", graph, queries, max(g["lo"] // 4, updates // count), deletes, entry=entry, scale=scale, **extra)
    del c["name"]
    return c
