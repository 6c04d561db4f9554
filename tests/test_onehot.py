"""Batches of queries on the tensor cores (tq_onehot.cu) against the CPU oracle,
bit for bit: ids and scores of the top k at the edges of its tiles (256 vectors,
32-query steps up to 192, 8 byte groups per stage, 256 per flush batch) and of
its lists (k up to 64, up to 256), with equal scores across tiles."""
import numpy as np
import pytest

import vectorcache_b200 as vcb
from oracle.oracle import Oracle
from vectorcache_b200.synthetic import power_law

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle():
    return Oracle()


def check(oracle, dim, bits, n, nq, k, tqplus=True, duplicates=False, order=None):
    db = power_law(n, dim, seed=11)
    if duplicates:
        db[n // 2:] = db[: n - n // 2]  # every score twice, far apart
    q = power_law(nq, dim, seed=12)
    if order == "ascending":  # scores grow along the index: thresholds stay low
        db = db[np.argsort(db @ q[0], kind="stable")]
    idx = vcb.TurboQuantIndex(dim, bits)
    if tqplus:
        idx.calibrate(db[:1000])
    idx.add(db)
    idx.prepare()
    res = idx.search(q, k)
    shift, scale = oracle.fit_calibration(db[:1000], bits) if tqplus else (None, None)
    packed, alpha = oracle.encode(db, bits, shift, scale)
    want_s, want_i = oracle.search_flat(q, bits, packed, alpha, k, shift, scale)
    assert np.array_equal(res.ids, want_i)
    assert np.array_equal(res.scores.view(np.uint32), want_s.view(np.uint32))
    idx.close()


@pytest.mark.parametrize("dim,bits,n,nq,k", [
    (8, 4, 16384, 32, 10),       # one part-full stage
    (24, 2, 16385, 33, 1),       # 6 byte groups, one vector in the last tile
    (64, 3, 20000, 192, 10),     # a full query tile
    (72, 4, 17000, 193, 10),     # two query tiles of 97 -> 128
    (264, 2, 16640, 40, 64),     # 66 groups: two groups in the last stage
    (520, 4, 16384, 64, 33),     # 260 groups: a flush batch of four
    (1024, 3, 16500, 5, 65),     # lists of 512 entries, five queries
    (136, 4, 40000, 385, 256),   # the largest k, three query tiles
])
def test_equals_the_oracle(oracle, dim, bits, n, nq, k):
    check(oracle, dim, bits, n, nq, k)


def test_equal_scores_keep_the_lower_ids(oracle):
    check(oracle, 64, 4, 18000, 36, 12, tqplus=False, duplicates=True)


@pytest.mark.parametrize("k", [10, 100])
def test_lists_that_overflow(oracle, k):
    check(oracle, 32, 4, 60000, 32, k, order="ascending")
