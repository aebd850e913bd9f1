"""The forms a round takes by size, against the CPU checker bit for bit."""
import numpy as np
import pytest

import octex_b200
from conftest import small_params

pytestmark = pytest.mark.gpu


def against_checker(oracle, idx, arrays, meta, queries, k, **kw):
    """Whole runs (nothing kept for inspection) against the checker, given the GPU's coordinates."""
    idx.set_debug(taps=True)
    apart = idx.search(queries, k, **kw)
    y = idx.fetch("y", np.uint16, (len(queries), -1))
    idx.set_debug()
    want_ids, want_dist, _ = oracle.Index(arrays, meta).search(queries, k, y_in=y, **kw)
    for dist, ids in (apart, idx.search(queries, k, **kw)):
        assert np.array_equal(ids, want_ids), (len(queries), kw)
        assert np.array_equal(dist.view(np.uint32), want_dist.view(np.uint32)), (len(queries), kw)


@pytest.mark.parametrize("distinct", [1, 3, 40, 4000])
def test_selection_among_equal_distances(oracle, distinct):
    """Rows that repeat: the bin of the last selected key holds any number of keys, more than are ranked
    aside (128) and all of them among these."""
    from octex_b200 import build_index, synth
    rng = np.random.default_rng(2)
    base = synth.plumbing(distinct, 48, seed=0)[rng.integers(0, distinct, 4000)]
    arrays, meta = build_index.build_arrays(base, small_params(table_len=32), device="cpu")
    idx = octex_b200.attach(arrays, meta, borrow=False)
    queries = synth.plumbing(40, 48, seed=1)
    for kw in (dict(read=16, starts=64, waves=2, rerank=40, wave_rerank=200), dict(read=16, starts=64, waves=1, sketch_rank=True)):
        against_checker(oracle, idx, arrays, meta, queries, 10, **kw)
    idx.close()
