"""GPU tests of what a captured graph bakes in: the scratch of the slot it was captured on, and the time limit."""
import numpy as np
import pytest

import csm
from csm import Batch
from helpers import small_workload
from oracle import Oracle

pytestmark = pytest.mark.gpu


def test_time_limit_set_after_the_capture():
    w = small_workload("c2", scale=0.05, nqueries=2)
    eng = csm.Engine(search_strategy=0, cuda_graphs=1)
    oracles = []
    for q in w.queries:
        eng.load_query(q)
        oracles.append(Oracle(q, w.data))
    eng.load_graph(w.data)
    a, b = w.batches[0], w.batches[1]
    n = min(len(a.src), len(b.src))
    cut = [Batch(x.src[:n], x.dst[:n], x.elabels[:n], x.is_delete[:n]) for x in (a, b, a, b)]
    for i, x in enumerate(cut):
        eng.set_time_limit(1 if i in (1, 2) else 0)
        rc, res = eng.apply_partial(x)
        full = [o.apply(x) for o in oracles]
        if i in (1, 2):
            assert rc == -4, "a 1-microsecond limit must stop the replayed launch"
        else:
            assert rc == 0
            assert [(r.positive, r.negative) for r in res] == [(f["pos"], f["neg"]) for f in full]
    assert eng.stats().graph_launches == len(cut)
    eng.close()


def test_tenants_with_graphs_move_between_slots():
    """Two tenants whose batches are replayed from graphs, on two slots: a tenant runs on either of them, and its
    graph has to use the slot's own control block and ring."""
    w = small_workload("c2", scale=0.02, nqueries=4)
    n = min(len(b.src) for b in w.batches)
    cut = [Batch(b.src[:n], b.dst[:n], b.elabels[:n], b.is_delete[:n]) for b in w.batches]
    undo = [Batch(b.src, b.dst, b.elabels, (1 - b.is_delete).astype(np.uint8)) for b in cut]
    steps = [x for _ in range(4) for pair in zip(cut, undo) for x in pair]
    engines, srv = [], csm.Server(slots=2)
    for part in (w.queries[:2], w.queries[2:]):
        e = csm.Engine(search_strategy=0, cuda_graphs=1, max_batch=n)
        for q in part:
            e.load_query(q)
        e.load_graph(w.data)
        e.apply(undo[0])  # captured on the engine's own scratch first
        srv.add_tenant(e)
        engines.append(e)
    oracles = [Oracle(q, w.data) for q in w.queries]
    for o in oracles:
        o.apply(undo[0])
    # Requests for one tenant alone, in between, change which slot each of the two runs on.
    requests = []
    for i, x in enumerate(steps):
        requests.append((srv.submit(x), x, [0, 1]))
        if i % 3 == 0:
            requests.append((srv.submit(x, tenant=i % 2), x, [i % 2]))
    for rid, x, tenants in requests:
        res = srv.wait(rid)[1]
        want = [oracles[2 * t + k].apply(x) for t in tenants for k in (0, 1)]
        assert [(r.positive, r.negative) for r in res] == [(f["pos"], f["neg"]) for f in want], f"request {rid}"
    assert all(e.stats().graph_launches > len(steps) for e in engines)
    srv.close()
    for e in engines:
        e.close()
