"""Delete by exact match over rows that agree in their first dimensions (padding, borders):
the same answers as by comparing whole rows, at a cost near that of rows that do not."""
import numpy as np
import pytest

from vann import workload

pytestmark = pytest.mark.gpu


def _index(vann_mod, base):
    n = len(base)
    idx = vann_mod.Index(base.shape[1], 8, 16, 1.2, capacity=n)
    idx.set_graph(base, np.zeros(n, np.uint32), np.zeros((n, 8), np.uint32), 0)
    return idx


# pairs left after a step above and below the block's list (512), whole rows equal, a tile of
# 64 queries and the remainder of one, 32 and 33 queries
@pytest.mark.parametrize("D,n,nq,head", [(8, 300, 70, 4), (8, 300, 70, 8), (128, 1000, 64, 40), (128, 700, 33, 128),
                                         (60, 260, 32, 56), (512, 500, 129, 256), (128, 300, 1, 124)])
def test_smallest_match_behind_equal_heads(vann_mod, D, n, nq, head):
    import torch

    rng = np.random.default_rng(D + n + head)
    base = rng.integers(0, 3, (n, D)).astype(np.float32)
    base[:, :head] = 1.0
    base[n // 2:] = base[: n - n // 2]  # each row twice
    idx = _index(vann_mod, base)
    dead = np.arange(0, n, 3)
    idx.delete(torch.from_numpy(dead.astype(np.int32)).cuda())
    q = base[rng.integers(0, n, nq)].copy()
    q[1::4, D - 1] += 5  # in no row
    buf = torch.zeros(nq * D + 1, device="cuda")  # queries off 16-byte alignment
    buf[1:] = torch.from_numpy(q.ravel()).cuda()
    got = idx.delete_by_vector(buf[1:].view(nq, D)).cpu().numpy()
    live = np.ones(n, bool)
    live[dead] = False
    first = {}
    for i in np.nonzero(live)[0]:
        first.setdefault(base[i].tobytes(), int(i))
    assert got.tolist() == [first.get(row.tobytes(), -1) for row in q]


def test_equal_heads_cost(vann_mod):
    """A thread per row and query, each stopping at its first difference, takes 8 times as
    long over rows whose first half is zero; whole-row comparisons by one thread took 59."""
    import torch

    ms = []
    for zero in (0, 64):
        base = workload.mixture(20000, 128, 20, seed=431)
        q = workload.mixture(500, 128, 20, seed=432)
        base[:, :zero] = 0
        q[:, :zero] = 0
        idx, qd = _index(vann_mod, base), torch.from_numpy(q).cuda()
        times = []
        for _ in range(12):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            try:
                idx.delete_by_vector(qd)
            except vann_mod.VannError as e:
                assert e.status == vann_mod.ERR_NOT_FOUND
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        ms.append(sorted(times[2:])[5])
    assert ms[1] < 8 * ms[0], ms
