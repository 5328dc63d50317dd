"""Plans rewritten after the planner — query edges that end in a leaf start once per data vertex of the
inner endpoint, and counting levels are settled from per-vertex sums although prefix vertices share
their label: the rewritten plans against the ones they stand for (CPU, native), and the engine
against the oracle on a graph whose hubs own many batch edges each."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import csm
from csm import DataGraph, QueryGraph, gen
from oracle import Oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gcsm-bu_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_rewritten_plans_count_what_the_edge_plans_count(tmp_path):
    exe = str(tmp_path / "leaf_group_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-o", exe,
                    os.path.join(ROOT, "tests", "native", "leaf_group_test.cpp"), os.path.join(CSRC, "plan.cpp"),
                    os.path.join(CSRC, "query.cpp"), "-I", CSRC], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.startswith("ok"), p.stdout + p.stderr


def query(labels, edges):
    s, d = zip(*edges)
    return QueryGraph(np.asarray(labels, dtype=np.uint32), np.array(s, dtype=np.uint32), np.array(d, dtype=np.uint32),
                      np.zeros(len(edges), dtype=np.uint32))


TRIANGLE_TAIL = [(0, 1), (1, 2), (1, 3), (2, 3)]
PATH6 = [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5)]
STAR = [(0, 1), (0, 2), (0, 3)]
QUERIES = [
    query([0, 1, 2, 2], TRIANGLE_TAIL),             # weighted: the leaf's label is its own
    query([1, 1, 0, 2], TRIANGLE_TAIL),             # weighted: only the inner endpoint shares it
    query([0, 1, 0, 0], TRIANGLE_TAIL),             # both, by the index of the updated edge
    query([2, 2, 0, 1, 0, 2], PATH6),               # a leaf in the tail next to another
    query([0, 1, 1, 1], STAR),                      # the counting level is the seed level
    query([0, 1, 2], [(0, 1), (1, 2)]),
    query([2, 2, 0, 1, 0, 3], PATH6),               # settled below vertices of the level's label
    query([1, 0, 1, 0, 3, 2], [(0, 1), (1, 2), (2, 3), (3, 4), (1, 5)]),  # and above another tail class
    query([1, 2, 0, 3, 1], [(0, 1), (1, 2), (2, 3), (3, 0), (2, 4)]),     # two pair intersections
    query([0, 1, 2, 3, 0], [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (2, 3), (0, 4)]),  # three lists of one vertex
    query([3, 3, 0, 1, 3, 0], [(0, 1), (0, 2), (2, 3), (3, 4), (4, 5)]),  # cut by a vertex of the tail's label
    query([0, 1, 0, 1, 1], [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (2, 3), (0, 4)]),  # of the prefix's labels
]


@pytest.mark.gpu
@pytest.mark.parametrize("strategy", [0, 1, 2, 3])
def test_rewritten_plans_equal_the_oracle(strategy):
    rng = np.random.default_rng(23)
    n = 400
    s, d = gen.chung_lu(n, 2400, 2.0, rng)          # uncapped: hubs with many batch edges
    vl = rng.integers(0, 4, size=n).astype(np.uint32)
    el = np.zeros(len(s), dtype=np.uint32)
    data, batches = gen.make_stream(n, s, d, el, rng, n_ins=240, n_del=240, batch=160)
    data = DataGraph(vl, data.src, data.dst, data.elabels)
    with csm.Engine(search_strategy=strategy, semi_bfs_items_per_warp=1) as eng:
        for q in QUERIES:
            eng.load_query(q)
        eng.load_graph(data)
        text = [eng.describe(i) for i in range(len(QUERIES))]
        assert "pendant counting level" in text[6] and "pendant counting level" in text[7]
        assert "pendant counting level" in text[10]
        assert any("counted per inner vertex" in t for t in text) and any("counted in the tail" in t for t in text)
        oracles = [Oracle(q, data) for q in QUERIES]
        seen = 0
        for b in batches:
            res = eng.apply(b)
            for qi, o in enumerate(oracles):
                r = o.apply(b)
                assert (res[qi].positive, res[qi].negative) == (r["pos"], r["neg"]), f"query {qi}"
                assert eng.edge_counts(qi) == (r["per_qe_pos"], r["per_qe_neg"]), f"query {qi} per-edge split"
                seen += r["pos"] * r["neg"] > 0
        assert seen > len(QUERIES)
