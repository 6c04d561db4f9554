"""Batches of queries on the tensor cores (tq_onehot.cu) against the CPU oracle,
bit for bit: ids and scores of the top k at the edges of its tiles (256 vectors,
32-query steps up to 192, 8 byte groups per stage, 256 per flush batch) and of
its lists (k up to 64, up to 256), with equal scores across tiles. Which batches
run there is an estimate (k > 32 from three queries on nearly always). Bucketed passes of at least 16 pairs per bucket against passes
small enough for the lookup scan."""
import numpy as np
import pytest

import vectorcache_b200 as vcb
from oracle.oracle import Oracle
from vectorcache_b200.synthetic import power_law, vmf_mixture

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
    (8, 4, 8192, 65, 10),        # the smallest index, one part-full stage
    (24, 2, 16385, 66, 1),       # 6 byte groups, one vector in the last tile
    (520, 3, 8449, 96, 10),      # 3-bit rows over two flush batches
    (1032, 4, 9000, 64, 33),     # 516 groups: three flush batches, the small-batch form
    (64, 3, 9000, 3, 40),        # three queries, 3-bit, the small-batch form
])
def test_equals_the_oracle(oracle, dim, bits, n, nq, k):
    check(oracle, dim, bits, n, nq, k)


def test_equal_scores_keep_the_lower_ids(oracle):
    check(oracle, 64, 4, 18000, 36, 12, tqplus=False, duplicates=True)
    check(oracle, 64, 4, 18000, 70, 12, tqplus=False, duplicates=True)


@pytest.mark.parametrize("k", [10, 100])
def test_lists_that_overflow(oracle, k):
    check(oracle, 32, 4, 60000, 32, k, order="ascending")


def test_many_queries_overflow_lists(oracle):
    check(oracle, 32, 4, 60000, 70, 10, order="ascending")


@pytest.mark.parametrize("dim,bits,n,k,n_probe,rerank_k", [
    (100, 4, 12000, 10, 24, 40),
    (51, 3, 12000, 7, 33, 0),      # dims padded to 56, 28 byte groups
    (48, 2, 12000, 64, 40, 0),     # 12 byte groups: less than two stages
    (520, 4, 6000, 10, 20, 0),     # two flush batches
    (64, 4, 12000, 1, 16, 0),      # a floor of one score
    # zero queries: every score equals the floor, more of them than a query's
    # region holds (4096 entries): the redo kernel.
    (64, 4, 12000, 1, 64, 0),
])
def test_bucketed_pass_equals_small_passes(dim, bits, n, k, n_probe, rerank_k):
    db = vmf_mixture(n, dim, seed=21, clusters=60)
    idx = vcb.BucketedTurboQuantIndex(dim, bits, vcb.BucketParams(
        n_probe=8, max_bucket_size=300, energy_soft=150, kmeans_iters=3, seed=7, rerank_k=rerank_k))
    idx.add(db)
    idx.prepare()
    nb = idx.info()["n_buckets"]
    nq = 16 * nb + 5  # every step holds at least 16 pairs per bucket
    q = np.random.default_rng(22).standard_normal((nq, dim)).astype(np.float32)
    if n_probe == 64:
        q[::5] = 0.0
    whole = idx.search(q, k, n_probe=n_probe)
    step = nb // 4  # probes 1..7 and the far ones stay below 16 pairs per bucket
    for s in range(0, min(nq, 8 * step), step):
        part = idx.search(q[s:s + step], k, n_probe=n_probe)
        assert np.array_equal(whole.ids[s:s + step], part.ids), s
        assert np.array_equal(whole.scores[s:s + step].view(np.uint32), part.scores.view(np.uint32)), s
    counts = (np.arange(nq) % n_probe + 1).astype(np.uint32)
    mixed = idx.search(q, k, n_probe=n_probe, n_probe_per_query=counts)
    rows = np.nonzero(counts == n_probe)[0]
    assert np.array_equal(mixed.ids[rows], whole.ids[rows])
    assert np.array_equal(mixed.scores[rows].view(np.uint32), whole.scores[rows].view(np.uint32))
    idx.close()


@pytest.mark.parametrize("n,nq,k", [
    (40_000, 1, 64),    # thousands of equal candidates: the merge's chunks
    (200_000, 1, 10),   # 980 of them: its sort
    (9_000, 1, 10),     # 50: no bound
    (60_000, 2, 256),
    (20_000, 70, 100),  # one-hot lists that every score enters
])
def test_zero_queries_return_the_lowest_ids(oracle, n, nq, k):
    db = power_law(n, 8, seed=31)
    q = np.zeros((nq, 8), np.float32)
    idx = vcb.TurboQuantIndex(8, 4)
    idx.add(db)
    idx.prepare()
    res = idx.search(q, k)
    packed, alpha = oracle.encode(db, 4, None, None)
    want_s, want_i = oracle.search_flat(q, 4, packed, alpha, k, None, None)
    assert np.array_equal(res.ids, want_i)
    assert np.array_equal(res.scores.view(np.uint32), want_s.view(np.uint32))
    idx.close()


def test_indexes_built_and_closed_by_several_threads():
    # Closed indexes' device blocks serve the next ones, across threads and streams.
    from concurrent.futures import ThreadPoolExecutor

    shapes = [(30_000, 64, 4, 5, 10), (50_000, 128, 3, 70, 10), (20_000, 256, 2, 3, 40)]

    def one(i):
        n, dim, bits, nq, k = shapes[i % 3]
        db, q = power_law(n, dim, seed=50 + i % 3), power_law(nq, dim, seed=60 + i % 3)
        idx = vcb.TurboQuantIndex(dim, bits)
        idx.calibrate(db[:2000])
        idx.add(db)
        idx.prepare()
        res = idx.search(q, k)
        idx.close()
        return res.ids, res.scores

    want = [one(i) for i in range(3)]
    with ThreadPoolExecutor(4) as pool:
        got = list(pool.map(one, range(12)))
    for i, (ids, scores) in enumerate(got):
        assert np.array_equal(ids, want[i % 3][0]), i
        assert np.array_equal(scores.view(np.uint32), want[i % 3][1].view(np.uint32)), i


@pytest.mark.parametrize("n_probe,k", [(9, 10), (10, 10), (10, 1), (14, 64)])
def test_lookup_step_after_a_onehot_step(n_probe, k):
    # Probes 1..7 have at least 16 pairs per bucket and the last step has not: it
    # appends to regions that the one-hot step may have filled. A zero query scores
    # every vector of seven buckets at its floor, more than the 4096 entries of its
    # region; its neighbours' regions, and the memory behind the last query's, have
    # to stay as they are.
    n, dim = 60000, 32
    db = vmf_mixture(n, dim, seed=23, clusters=60)
    idx = vcb.BucketedTurboQuantIndex(dim, 4, vcb.BucketParams(
        n_probe=8, max_bucket_size=4000, energy_soft=2000, kmeans_iters=3, seed=7))
    idx.add(db)
    idx.prepare()
    nb = idx.info()["n_buckets"]
    sizes = idx.layout()["bucket_size"]
    assert sizes[1:8].sum() > 4096  # a zero query's first probes: equal scores, lowest ids
    nq = 5 * nb // 2
    assert 7 * nq >= 16 * nb > (n_probe - 8) * nq
    q = np.random.default_rng(24).standard_normal((nq, dim)).astype(np.float32)
    q[::3] = 0.0
    q[-1] = 0.0
    whole = idx.search(q, k, n_probe=n_probe)
    for s in range(0, nq, nb):  # 7 nb pairs: every step on the lookup scan
        part = idx.search(q[s:s + nb], k, n_probe=n_probe)
        assert np.array_equal(whole.ids[s:s + nb], part.ids), s
        assert np.array_equal(whole.scores[s:s + nb].view(np.uint32), part.scores.view(np.uint32)), s
    idx.close()


@pytest.mark.parametrize("nb_queries,many", [(4, 4), (4, 1), (16, 1)])
def test_probe_counts_per_query_decide_by_their_pairs(nb_queries, many):
    # One query in `many` has 40 probes, the others 9: the steps' bounds allow the
    # one-hot scan, their pairs do for some steps only (few pairs: the lookup scan).
    idx = vcb.BucketedTurboQuantIndex(64, 4, vcb.BucketParams(
        n_probe=8, max_bucket_size=300, energy_soft=150, kmeans_iters=3, seed=7))
    idx.add(vmf_mixture(12000, 64, seed=25, clusters=60))
    idx.prepare()
    nb = idx.info()["n_buckets"]
    nq = nb_queries * nb
    q = np.random.default_rng(26).standard_normal((nq, 64)).astype(np.float32)
    counts = np.where(np.arange(nq) % many == 0, 40, 9).astype(np.uint32)
    whole = idx.search(q, 10, n_probe=40, n_probe_per_query=counts)
    step = nb // 4
    for s in range(0, nq, step):
        part = idx.search(q[s:s + step], 10, n_probe=40, n_probe_per_query=counts[s:s + step])
        assert np.array_equal(whole.ids[s:s + step], part.ids), s
        assert np.array_equal(whole.scores[s:s + step].view(np.uint32), part.scores.view(np.uint32)), s
    idx.close()


@pytest.mark.parametrize("n,nq,k", [
    (2048, 3, 1), (2048, 2, 32),   # one list: fewer candidates than lanes, as many
    (16384, 1, 32), (16385, 2, 32), (18433, 1, 29),
    (65536, 1, 8), (65537, 1, 8),  # 256 candidates: the most that one warp merges; one list more
    (65536, 2, 9),                 # the first k of the CTA's merge
    (524288, 1, 1), (524289, 1, 1),
])
@pytest.mark.parametrize("zeros", [False, True])
def test_merge_of_few_candidates(oracle, n, nq, k, zeros):
    db = power_law(n, 8, seed=33)
    q = np.zeros((nq, 8), np.float32) if zeros else power_law(nq, 8, seed=34)
    idx = vcb.TurboQuantIndex(8, 4)
    idx.add(db)
    idx.prepare()
    res = idx.search(q, k)
    packed, alpha = oracle.encode(db, 4, None, None)
    want_s, want_i = oracle.search_flat(q, 4, packed, alpha, k, None, None)
    assert np.array_equal(res.ids, want_i)
    assert np.array_equal(res.scores.view(np.uint32), want_s.view(np.uint32))
    idx.close()


@pytest.mark.parametrize("dim,bits,n,nq,k", [
    (24, 2, 40001, 200, 1),      # 6 byte groups, one vector in the last tile, k = 1
    (64, 3, 50000, 130, 3),
    (8, 4, 100000, 66, 32),
    (8, 4, 8192, 66, 1),         # the lookup scan: the smallest batch and k above 64 queries
    (64, 3, 16384, 66, 3),
    (768, 2, 8192, 600, 1),
])
def test_batches_above_64_queries_equal_the_oracle(oracle, dim, bits, n, nq, k):
    check(oracle, dim, bits, n, nq, k)
