"""A kernel that gave up waiting sets its owner's status word. Here the test sets the
word itself, as such a kernel would: the call that waits for the work reports it,
once, and no other call does."""
import ctypes as C

import numpy as np
import pytest

import vectorcache_b200 as vcb
from vectorcache_b200.multi import MultiIndex
from vectorcache_b200.synthetic import power_law, vmf_mixture

pytestmark = pytest.mark.gpu


def _word(name, handle, *args):
    fn = getattr(vcb.load_library(), name)
    fn.restype = C.POINTER(C.c_uint32)
    fn.argtypes = [C.c_void_p] + [C.c_size_t] * len(args)
    return fn(handle, *args)


def _gave_up(call):
    with pytest.raises(vcb.TurboQuantError, match="gave up waiting") as e:
        call()
    assert e.value.code == vcb.TQ_ERR_CUDA


@pytest.fixture(scope="module")
def flat():
    db = power_law(20_000, 64, seed=41)
    idx = vcb.TurboQuantIndex(64, 4)
    idx.add(db)
    idx.prepare()
    yield idx, db
    idx.close()


def test_host_and_queued_searches_report_their_own(flat):
    idx, db = flat
    call, queued = _word("tq_test_index_status", idx._h, 0), _word("tq_test_index_status", idx._h, 1)
    want = idx.search(db[:70], 5).ids
    queued[0] = 1  # a search_device that gave up
    assert np.array_equal(idx.search(db[:70], 5).ids, want)
    _gave_up(idx.synchronize)
    idx.synchronize()
    call[0] = 1
    _gave_up(lambda: idx.search(db[:70], 5))
    idx.synchronize()
    assert np.array_equal(idx.search(db[:70], 5).ids, want)


def test_multi_index_launch_reports_at_synchronize(flat):
    torch = pytest.importorskip("torch")
    idx, db = flat
    multi = MultiIndex([idx, idx])
    multi.plan([80, 3], [5, 5], autotune=True)
    word = _word("tq_test_multi_status", multi._h)
    for stream in (None, torch.cuda.Stream()):
        multi.set_queries(0, db[:80])
        multi.set_queries(1, db[:3])
        multi.launch(stream)
        multi.synchronize()
        assert np.array_equal(multi.results(0)[1], idx.search(db[:80], 5).ids)
        word[0] = 1
        assert idx.search(db[:80], 5).ids.shape == (80, 5)
        idx.synchronize()
        _gave_up(multi.synchronize)
        multi.synchronize()
    multi.close()


def test_served_batches_report_to_their_requests():
    idx = vcb.BucketedTurboQuantIndex(32, 4, vcb.BucketParams(n_probe=8, max_bucket_size=300, energy_soft=150, seed=7))
    db = vmf_mixture(6_000, 32, seed=42, clusters=20)
    idx.add(db)
    idx.prepare()
    srv = vcb.Server(hbm_budget_bytes=20 << 30, max_slots=1, max_batch=64)
    target = srv.add_bucketed(idx, max_k=10, max_probe=16)
    srv.start()
    want = idx.search(db[:8], 10, n_probe=16).ids
    word = _word("tq_test_server_status", srv._h, 0)
    word[0] = 1
    req = srv.submit(target, db[:8], 10, n_probe=16)
    _gave_up(req.wait)
    assert np.array_equal(idx.search(db[:8], 10, n_probe=16).ids, want)
    assert np.array_equal(srv.submit(target, db[:8], 10, n_probe=16).wait()[1], want)
    srv.close()
    idx.close()
