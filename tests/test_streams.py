"""The engine's and the slots' streams do not wait for the default stream, so what their kernels read must not be
written through it: a copy from pageable memory or a fill there may still be on its way when the kernel starts."""
import glob
import os
import re
import threading

import numpy as np
import pytest

import csm
from csm import Batch, DataGraph, QueryGraph
from helpers import random_graph
from oracle import Oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_writes_through_the_default_stream():
    found = []
    for path in glob.glob(os.path.join(ROOT, "gcsm-bu_b200", "csrc", "*.c*")):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"\bcudaMemset\s*\(|\bcudaMemcpy\s*\([^;]*cudaMemcpyHostToDevice", text):
            found.append(f"{os.path.basename(path)}: {m.group(0)[:60]}")
    assert not found, found


@pytest.mark.gpu
@pytest.mark.parametrize("snapshot", [False, True])
def test_loads_beside_other_copies(tmp_path, snapshot):
    """Loads while another stream keeps the copy engines busy, so that copies arrive late."""
    import torch
    rng = np.random.default_rng(4)
    vl, s, d, el = random_graph(4000, 60000, 4, rng, nel=4)
    data = DataGraph(vl, s, d, el)
    q = QueryGraph(np.array([0, 1, 2, 1], np.uint32), np.array([0, 1, 2], np.uint32), np.array([1, 2, 3], np.uint32),
                   np.array([0, 1, 0], np.uint32))
    pick = rng.permutation(len(s))[:2000]
    batches = [Batch(s[pick], d[pick], el[pick], np.ones(2000, np.uint8)), Batch(s[pick], d[pick], el[pick])]
    want = []
    oracle = Oracle(q, data)
    for b in batches:
        r = oracle.apply(b)
        want.append((r["pos"], r["neg"]))
    assert want[0][1] > 0
    path = str(tmp_path / "g.snap")
    with csm.Engine(max_batch=2048, frontier_bytes=1 << 20) as eng:
        eng.load_query(q)
        eng.load_graph(data)
        eng.save_snapshot(path)
    src = torch.empty(64 << 20, dtype=torch.uint8, pin_memory=True)
    dst = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    side, stop = torch.cuda.Stream(), threading.Event()

    def busy():
        with torch.cuda.stream(side):
            while not stop.is_set():
                for _ in range(8):
                    dst.copy_(src, non_blocking=True)
                side.synchronize()

    t = threading.Thread(target=busy)
    t.start()
    try:
        for _ in range(12):
            with csm.Engine(max_batch=2048, frontier_bytes=1 << 20) as eng:
                eng.load_query(q)
                if snapshot:
                    eng.load_snapshot(path)
                else:
                    eng.load_graph(data)
                got = [eng.apply(b)[0] for b in batches]
            assert [(r.positive, r.negative) for r in got] == want
    finally:
        stop.set()
        t.join()
