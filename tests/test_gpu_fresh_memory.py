"""List slots past a node's degree hold what the device memory held before the index: no
search may use them.  Inserted nodes never had theirs written."""
import numpy as np
import pytest

from vann import workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,L", [(32, 16), (64, 48), (64, 200), (128, 100)])
def test_small_searches_after_inserts(vann_mod, R, L):
    import torch

    n, m, D = 800, 700, 32
    base = workload.mixture(n + m, D, 12, seed=411)
    rows = torch.from_numpy(base).cuda()
    q = torch.from_numpy(workload.mixture(40, D, 12, seed=412)).cuda()
    got = []
    for fill in (0, -1):  # what the index's memory holds at first
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held = [torch.full((4 << 20,), fill, dtype=torch.int32, device="cuda") for _ in range(16)]
        torch.cuda.synchronize()
        del held
        torch.cuda.empty_cache()  # given back: the index's allocations reuse it
        idx = vann_mod.Index(D, R, 48, 1.2, capacity=n + m)
        idx.build(rows[:n], batch=0, seed=5)
        for at in range(n, n + m, 100):
            idx.insert(rows[at: at + 100])
        ids, d, st = idx.search_stats(q, k=10, L=L)
        got.append((ids.cpu(), d.cpu(), st.cpu()))
        idx.sync()
        assert int((idx.get_graph()[1] < R).sum()) > 0  # lists with such slots
        idx.close()
    assert all(torch.equal(x, y) for x, y in zip(*got))
    assert np.mean([i >= n for i in got[0][0].numpy().ravel()]) > 0.2  # inserted rows are found
