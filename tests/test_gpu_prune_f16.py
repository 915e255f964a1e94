"""RobustPrune on float rows (prune_tc.cu): a tensor-core Gram matrix of f16 rows as a
filter, FP32 distances where it cannot decide.  Builds against the oracle at the edges of
its passes, and the FP32 decisions pinned bit for bit."""
import numpy as np
import pytest

from vann import workload

pytestmark = pytest.mark.gpu


def _rows_equal(deg_a, adj_a, deg_b, adj_b):
    return [i for i in range(len(deg_a)) if not np.array_equal(adj_a[i, :deg_a[i]], adj_b[i, :deg_b[i]])]


@pytest.mark.parametrize("D,R,L,max_visited", [(4, 8, 32, 600), (12, 32, 75, 600), (64, 64, 100, 128), (100, 48, 64, 64),
                                               (128, 1, 20, 600), (128, 128, 130, 600), (128, 64, 260, 600)])
def test_build_and_insert_match_oracle(oracle, vann_mod, D, R, L, max_visited):
    """Integer rows (every distance exact, so the oracle's sequential sums have the same
    bits) without a uint8 copy: candidate counts below, around and above 128 and 256,
    lists cut at max_visited, rows whose length is not a multiple of 8."""
    import torch

    n, n1 = 1500, 203
    base = workload.mixture(n + n1, D, 15, seed=151)
    deg0, adj0 = oracle.random_graph(n, R, 9)
    deg = np.zeros(n + n1, np.uint32)
    adj = np.zeros((n + n1, R), np.uint32)
    deg[:n], adj[:n] = deg0, adj0
    og = oracle.Graph(base, deg, adj)
    entry = oracle.medoid(base[:n])
    for first, count, skip in ((0, n, 2), (n, n1, 0)):
        assert og.vamana_batch(first, count, L, 1.2, entry, max_visited=max_visited, skip_mode=skip,
                               bloom_mode=oracle.BLOOM_SNAPSHOT) == 0
    idx = vann_mod.Index(D, R, L, 1.2, capacity=n + n1, max_visited=max_visited)
    idx.build(torch.from_numpy(base[:n]).cuda(), batch=0, seed=9)
    idx.insert(torch.from_numpy(base[n:]).cuda())
    _, gdeg, gadj = idx.get_graph()
    assert _rows_equal(gdeg, gadj, og.deg, og.adj) == []


def _dist_f32(x, y):
    """FP32 squared distances of rows x [a, D] to rows y [b, D] in the kernels' order:
    16 lanes of 8 dimensions, even and odd dimensions accumulated apart by fused
    multiply-adds, the lanes added pairwise (t with t ^ 8, ^ 4, ^ 2, ^ 1).  Each fused
    step is exact in FP64 before its rounding (integer rows below 2^13)."""
    D = x.shape[1]
    d = np.zeros((len(x), len(y), 128))
    d[:, :, :D] = y[None].astype(np.float64) - x[:, None].astype(np.float64)
    d = d.reshape(len(x), len(y), 16, 4, 2)
    acc = np.zeros((len(x), len(y), 16, 2), np.float32)
    for p in range(4):
        acc = (d[:, :, :, p] * d[:, :, :, p] + acc.astype(np.float64)).astype(np.float32)
    v = acc[..., 0] + acc[..., 1]
    for off in (8, 4, 2, 1):
        v = v[..., :off] + v[..., off:2 * off]
    return v[..., 0]


@pytest.mark.parametrize("alpha", [1.0, 1.2])
@pytest.mark.parametrize("D,R,n_dead", [(4, 16, 2), (64, 32, 2), (100, 64, 2), (128, 128, 1), (128, 128, 2), (128, 128, 3)])
def test_decisions_have_the_kernels_fp32_order(vann_mod, D, R, n_dead, alpha):
    """Consolidation of a set graph whose rows make FP32 sums round (values to +-4000):
    every re-pruned list equals a plain restatement with the same summation order.  With
    alpha = 1 and distances this close together many pairs fall to the FP32 step."""
    import torch

    rng = np.random.default_rng(5 + D + n_dead)
    n, alpha = 500, np.float32(alpha)
    base = rng.integers(-4000, 4001, (n, D)).astype(np.float32)
    dead = list(range(n - n_dead, n))
    deg = np.full(n, R, np.uint32)
    deg[: n // 2] = rng.integers(max(1, R // 2), R + 1, n // 2)
    adj = np.stack([rng.permutation(n - n_dead)[:R] for _ in range(n)]).astype(np.uint32)
    hit = list(range(0, 180, 7))  # 26 nodes: the last pass alone
    for p in hit:  # these nodes point at deleted ones
        for j, x in enumerate(dead):
            adj[p, (7 * p + 5 * j) % deg[p]] = x
    idx = vann_mod.Index(D, R, 64, float(alpha), capacity=n)
    idx.set_graph(base, deg, adj, entry=100)
    idx.delete(torch.tensor(dead, dtype=torch.int32, device="cuda"))
    idx.consolidate()
    _, gdeg, gadj = idx.get_graph()
    cap = min(2048, max(600, 2 * R))
    sizes = []
    for p in hit:
        cand = []
        for x in adj[p, : deg[p]]:
            cand += [int(x)] if x not in dead else [int(u) for u in adj[x, : deg[x]]]
        cand = [c for c in dict.fromkeys(cand) if c != p and c not in dead][:cap]
        sizes.append(len(cand))
        d = _dist_f32(base[p:p + 1], base[cand])[0]
        order = np.argsort(d, kind="stable")
        cand, d = np.array(cand)[order], d[order]
        pair = _dist_f32(base[cand], base[cand])
        live, chosen = np.ones(len(cand), bool), []
        for t in range(len(cand)):
            if live[t] and len(chosen) < R:
                chosen.append(cand[t])
                live &= ~(pair[t] * alpha <= d)
        assert gadj[p, : gdeg[p]].tolist() == chosen, p
    assert max(sizes) > R


def test_float_rows_build_the_same_graph_beside_an_inexact_copy(vann_mod):
    """Float rows with and without a (fitted, inexact) uint8 copy give the same graph."""
    import torch

    base = torch.from_numpy(workload.mixture(4000, 96, 20, seed=152, sigma=0.05, integer=False, unit_norm=True)).cuda()
    got = []
    for stores in (("f32",), ("f32", "u8")):
        idx = vann_mod.Index(96, 64, 100, 1.2, capacity=4000, stores=stores)
        idx.build(base, batch=1000, seed=3)
        assert idx.info()["pruned_tc"] == 0 and idx.info()["pruned_cuda"] >= 4000
        got.append(idx.get_graph())
    assert _rows_equal(got[0][1], got[0][2], got[1][1], got[1][2]) == []


@pytest.mark.parametrize("scale", [1e-18, 1.0, 1e17])
def test_rows_of_extreme_magnitude_and_duplicates(vann_mod, scale):
    """The same lists at any scale of the rows (powers of two scale FP32 sums exactly; far
    from 1 the filter stands back for the FP32 distances), with duplicate rows among them."""
    import torch

    rng = np.random.default_rng(17)
    base = rng.integers(-3, 4, (900, 32)).astype(np.float32)
    base[300:360] = base[0]  # duplicates
    s = np.float32(2.0 ** round(np.log2(scale)))
    got = []
    for f in (np.float32(1.0), s):
        idx = vann_mod.Index(32, 24, 60, 1.25, capacity=900)
        idx.build(torch.from_numpy(base * f).cuda(), batch=300, seed=3, entry=5)
        got.append(idx.get_graph())
    assert _rows_equal(got[0][1], got[0][2], got[1][1], got[1][2]) == []
