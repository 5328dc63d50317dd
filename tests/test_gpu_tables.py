"""GPU tests of the counting tables an engine keeps: their size follows the graph's."""
import ctypes

import numpy as np
import pytest

import csm
from csm import DataGraph
from helpers import cycle, random_graph
from oracle import Oracle

pytestmark = pytest.mark.gpu


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
