"""GPU tests of the embedding rows a batch hands out (csm_config.materialize_rows)."""
import numpy as np
import pytest

import csm
from csm import Batch
from helpers import small_workload
from oracle import Oracle

pytestmark = pytest.mark.gpu


def test_rows_are_those_of_the_last_batch():
    """A batch without deletions, or without updates, leaves no rows of the batches before it."""
    w = small_workload("c1", scale=0.2)
    eng = csm.Engine(materialize_rows=1 << 16)
    eng.load_query(w.queries[0])
    eng.load_graph(w.data)
    oracle = Oracle(w.queries[0], w.data)
    none = np.zeros(0, dtype=np.uint32)
    seen = 0
    for b in w.batches[:3]:
        ones = np.ones(len(b.src), dtype=np.uint8)
        for step in (Batch(b.src, b.dst, b.elabels), Batch(b.src, b.dst, b.elabels, ones),
                     Batch(b.src, b.dst, b.elabels), Batch(b.src, b.dst, b.elabels, 0 * ones),
                     Batch(b.src, b.dst, b.elabels, ones), Batch(none, none, none)):
            res = eng.apply(step)[0]
            r = oracle.apply(step, rows=True)
            assert (res.positive, res.negative) == (r["pos"], r["neg"])
            for sign, count in ((1, res.positive), (-1, res.negative)):
                got = eng.embeddings(0, sign)
                assert len(got) == count
                assert np.array_equal(got, oracle.rows(sign))
            seen += res.negative
    eng.close()
    assert seen > 0
