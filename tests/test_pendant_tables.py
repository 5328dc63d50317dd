"""Pendant tables of an engine: which plans get one (CPU, native), and an engine with more pendant counting levels
than tables against the oracle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import csm
from csm import Batch, DataGraph, QueryGraph
from helpers import random_graph
from oracle import Oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gcsm-bu_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_which_plans_get_a_table(tmp_path):
    exe = str(tmp_path / "pendant_tables_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-o", exe,
                    os.path.join(ROOT, "tests", "native", "pendant_tables_test.cpp"), os.path.join(CSRC, "plan.cpp"),
                    os.path.join(CSRC, "query.cpp"), "-I", CSRC], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0 and p.stdout.startswith("ok"), p.stdout + p.stderr


def path(labels):
    n = len(labels)
    return QueryGraph(np.array(labels, dtype=np.uint32), np.arange(n - 1, dtype=np.uint32), np.arange(1, n, dtype=np.uint32),
                      np.zeros(n - 1, dtype=np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("strategy", [0, 2])
def test_more_pendant_levels_than_tables(strategy):
    rng = np.random.default_rng(11)
    vl, s, d, el = random_graph(600, 5000, 6, rng)
    # Paths with a label that returns, and at the end one that is pendant as it stands.
    queries = [path([a, b, c, a if i % 2 else b, e]) for i, (a, b, c, e) in
               enumerate(rng.permutation(6)[:4].tolist() for _ in range(14))] + [path([0, 1, 2, 3, 4])]
    keep = 4000
    data = DataGraph(vl, s[:keep], d[:keep], el[:keep])
    with csm.Engine(search_strategy=strategy, semi_bfs_items_per_warp=1) as eng:
        for q in queries:
            eng.load_query(q)
        eng.load_graph(data)
        text = [eng.describe(i) for i in range(len(queries))]
        assert sum(t.count("pendant counting level") for t in text) > 16
        assert any("without a table" in t for t in text) and "without a table" not in text[-1]
        assert "pendant counting level" in text[-1]
        oracles = [Oracle(q, data) for q in queries]
        pick = rng.permutation(len(s))[:900]
        seen = 0
        for part in np.array_split(pick, 3):
            b = Batch(s[part], d[part], el[part], (part < keep).astype(np.uint8))
            res = eng.apply(b)
            for qi, o in enumerate(oracles):
                r = o.apply(b)
                assert (res[qi].positive, res[qi].negative) == (r["pos"], r["neg"]), f"query {qi}"
                seen += r["pos"] > 0 and r["neg"] > 0
        assert seen > len(queries)
