"""Device blocks that closed indexes leave for later allocations: giving one back
does not disturb a graph that another thread captures, and trim() hands them to
the rest of the process."""
import threading

import pytest

import vectorcache_b200 as vcb
from vectorcache_b200.synthetic import power_law

pytestmark = pytest.mark.gpu


def _index(n, dim):
    db = power_law(n, dim, seed=5)
    idx = vcb.TurboQuantIndex(dim, 4)
    idx.add(db)
    idx.prepare()
    return idx, db


def test_an_index_closes_while_another_thread_captures():
    torch = pytest.importorskip("torch")
    idx, db = _index(40_000, 128)  # 2.5 MB of codes: a block the cache keeps
    idx.search(db[:4], 10)
    x = torch.ones(1024, device="cuda")
    y = torch.zeros(1024, device="cuda")
    x * 2 + 1  # kernels loaded
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        y.copy_(x * 2)
        t = threading.Thread(target=idx.close)
        t.start()
        t.join()
        y.add_(1)
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert bool((y == 3).all())
    again, db = _index(40_000, 128)
    assert (again.search(db[:4], 1).ids[:, 0] == range(4)).all()
    again.close()


def test_trim_gives_kept_blocks_back():
    torch = pytest.importorskip("torch")
    vcb.trim()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    idx, _ = _index(400_000, 128)  # 205 MB of rows until prepare(), 25.6 MB of codes
    idx.close()
    kept = before - torch.cuda.mem_get_info()[0]
    vcb.trim()
    assert kept >= 200 << 20
    assert before - torch.cuda.mem_get_info()[0] <= 8 << 20
    assert vcb.trim() is None  # nothing left: no error
