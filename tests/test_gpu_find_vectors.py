"""Delete by exact match: smallest live id per query over row and query counts around the
kernel's blocks, duplicate rows past its pair list, rows that agree in their head only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,n,nq", [(4, 1, 1), (12, 255, 65), (128, 257, 64), (100, 3000, 700), (4, 2000, 300)])
def test_smallest_live_match(vann_mod, D, n, nq):
    import torch

    rng = np.random.default_rng(D + n)
    hi = 2 if D == 4 else 4  # few values: many duplicates and many equal heads
    base = rng.integers(0, hi, (n, D)).astype(np.float32)
    if D > 4:
        base[:, :4] = rng.integers(0, 2, (n, 4))
        base[n // 2:] = base[: n - n // 2]
    idx = vann_mod.Index(D, 8, 16, 1.2, capacity=n)
    deg, adj = np.zeros(n, np.uint32), np.zeros((n, 8), np.uint32)
    idx.set_graph(base, deg, adj, 0)
    dead = np.arange(0, n, 5)[1:] if n > 5 else np.array([], np.int64)
    if len(dead):
        idx.delete(torch.from_numpy(dead.astype(np.int32)).cuda())
    q = base[rng.integers(0, n, nq)].copy()
    q[::9, D - 1] += 7  # in no row
    got = idx.delete_by_vector(torch.from_numpy(q).cuda()).cpu().numpy()
    live = np.ones(n, bool)
    live[dead] = False
    first = {}
    for i in np.nonzero(live)[0]:
        first.setdefault(base[i].tobytes(), int(i))
    assert got.tolist() == [first.get(row.tobytes(), -1) for row in q]
