"""The multi-index autotuner may send every batch to the single-index kernels, and
times them on queries like real ones (zero queries make every score equal the
threshold: the one-hot scan then looked many times slower than it is)."""
import numpy as np
import pytest

import vectorcache_b200 as vcb
from vectorcache_b200.multi import MultiIndex
from vectorcache_b200.synthetic import power_law

pytestmark = pytest.mark.gpu


def test_equal_heavy_batches_are_all_direct():
    db = power_law(100_000, 256, seed=61)
    indexes = []
    for part in (db[:50_000], db[50_000:]):
        idx = vcb.TurboQuantIndex(256, 4)
        idx.add(part)
        idx.prepare()
        indexes.append(idx)
    multi = MultiIndex(indexes)
    multi.plan([300, 300], [10, 10], autotune=True)
    assert multi.config()["direct_indexes"] == 2
    multi.launch()
    multi.synchronize()
    want = indexes[1].search(np.zeros((300, 256), np.float32), 10)
    assert np.array_equal(multi.results(1)[1], want.ids)  # planning leaves zero queries behind
    q = power_law(300, 256, seed=62)
    for i in range(2):
        multi.set_queries(i, q)
    multi.launch()
    multi.synchronize()
    for i, idx in enumerate(indexes):
        want = idx.search(q, 10)
        got_s, got_i = multi.results(i)
        assert np.array_equal(got_i, want.ids)
        assert np.array_equal(got_s.view(np.uint32), want.scores.view(np.uint32))
    multi.close()
    for idx in indexes:
        idx.close()
