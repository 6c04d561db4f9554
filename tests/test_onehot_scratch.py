"""Device scratch of one-hot batches: passes stay within their bound and change no
result."""
import numpy as np
import pytest

import vectorcache_b200 as vcb
from vectorcache_b200.synthetic import power_law

pytestmark = pytest.mark.gpu


def test_a_large_batch_runs_in_bounded_passes():
    # 40,000 queries of k = 256: 1.1 KB per list, 25 ranges and more, about 4.5 GB of
    # published lists in one pass; 1 GiB is the bound, 32,768 queries another.
    torch = pytest.importorskip("torch")
    n, dim, k = 30_000, 8, 256
    db = power_law(n, dim, seed=51)
    idx = vcb.TurboQuantIndex(dim, 4)
    idx.add(db)
    idx.prepare()
    q = torch.from_numpy(power_law(40_000, dim, seed=52)).cuda()
    scores = torch.empty((40_000, k), device="cuda")
    ids = torch.empty((40_000, k), dtype=torch.int64, device="cuda")
    vcb.trim()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    idx.search_device(q, k, scores, ids)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 3 << 29  # the lists, the running lists, LUTs
    for at in (0, 191, 9_000, 20_000, 32_760, 39_900):
        part = idx.search(q[at:at + 100].cpu().numpy(), k)
        assert np.array_equal(ids[at:at + 100].cpu().numpy().astype(np.uint64), part.ids), at
        assert np.array_equal(scores[at:at + 100].cpu().numpy().view(np.uint32), part.scores.view(np.uint32)), at
    idx.close()
