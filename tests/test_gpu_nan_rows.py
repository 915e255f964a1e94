"""Rows with a NaN in them sort behind every other row: a search over an index that holds
some gives what it gives when those rows are infinitely far away instead."""
import numpy as np
import pytest

from vann import workload

pytestmark = pytest.mark.gpu

N, BAD = 900, 150


def _graphs(vann_mod, D, R, stores):
    """Two indexes over one graph: every tenth row NaN in one, of distance +inf in the other."""
    import torch

    base = workload.mixture(N, D, 12, seed=401)
    idx = vann_mod.Index(D, R, 48, 1.2, capacity=N)
    idx.build(torch.from_numpy(base).cuda(), batch=0, seed=5)
    entry = idx.info()["entry"]
    _, deg, adj = idx.get_graph()
    rng = np.random.default_rng(7)
    bad = np.setdiff1d(rng.permutation(N), [entry], assume_unique=True)[:BAD]
    out = []
    for value in (np.nan, 3e38):
        rows = base.copy()
        rows[bad, 1] = value
        i = vann_mod.Index(D, R, 48, 1.2, capacity=N, stores=stores)
        i.set_graph(rows, deg, adj, entry)
        out.append(i)
    return out, bad


def _same(vann_mod, pair, bad, nq, D, **kw):
    import torch

    q = torch.from_numpy(workload.mixture(nq, D, 12, seed=402)).cuda()
    (ids, d, st), (ids2, d2, st2) = (i.search_stats(q, **kw) for i in pair)
    assert torch.equal(ids, ids2) and torch.equal(st, st2)
    far = torch.isin(ids, torch.from_numpy(bad.astype(np.int32)).cuda())
    assert bool(torch.isnan(d[far]).all()) and bool(torch.isinf(d2[far]).all())
    assert torch.equal(d[~far], d2[~far])
    return far


@pytest.mark.parametrize("D,R,L,store,rerank", [(32, 32, 100, "f32", False), (128, 64, 65, "bf16", True),
                                                (32, 64, 1000, "f32", False), (128, 96, 40, "f32", False),
                                                (160, 64, 300, "f32", True), (384, 20, 40, "bf16", False)])
def test_warp_per_query_lists(vann_mod, D, R, L, store, rerank):
    import torch

    nq = 7 * torch.cuda.get_device_properties(0).multi_processor_count + 64  # too many for a CTA per query
    pair, bad = _graphs(vann_mod, D, R, ("f32", store) if store != "f32" else ("f32",))
    far = _same(vann_mod, pair, bad, nq, D, k=L, L=L, store=store, rerank=rerank)
    assert L < 1000 or bool(far.any())  # long lists reach the far rows


@pytest.mark.parametrize("D,R,L,store", [(32, 32, 100, "f32"), (128, 64, 130, "f32"), (128, 64, 48, "bf16"),
                                         (128, 128, 20, "f32"), (160, 64, 256, "bf16")])
def test_cta_per_query(vann_mod, D, R, L, store):
    """Small batches: as with the far rows at +inf, and as the same queries in a large batch."""
    import torch

    pair, bad = _graphs(vann_mod, D, R, ("f32", store) if store != "f32" else ("f32",))
    _same(vann_mod, pair, bad, 40, D, k=L, L=L, store=store)
    nq = 7 * torch.cuda.get_device_properties(0).multi_processor_count + 64
    q = torch.from_numpy(workload.mixture(nq, D, 12, seed=402)).cuda()
    few, all_ = (pair[0].search_stats(q[:c].contiguous(), k=L, L=L, store=store) for c in (40, nq))
    assert torch.equal(few[0], all_[0][:40]) and torch.equal(few[2], all_[2][:, :40])
    assert torch.equal(few[1].view(torch.int32), all_[1][:40].view(torch.int32))


@pytest.mark.parametrize("L", [1, 12, 64, 100])
def test_nan_entry_and_nan_query(vann_mod, L):
    """An entry row with a NaN stays behind every other entry; a query with one ends at once."""
    import torch

    base = workload.mixture(N, 64, 12, seed=403)
    idx = vann_mod.Index(64, 32, 48, 1.2, capacity=N)
    idx.build(torch.from_numpy(base).cuda(), batch=0, seed=5)
    _, deg, adj = idx.get_graph()
    rows = base.copy()
    rows[3, 0] = np.nan
    idx.set_graph(rows, deg, adj, 3)
    nq = 7 * torch.cuda.get_device_properties(0).multi_processor_count + 64
    q = torch.from_numpy(workload.mixture(nq, 64, 12, seed=404)).cuda()
    q[5, 9] = float("nan")
    few, all_ = (idx.search_stats(q[:c].contiguous(), k=L, L=L) for c in (40, nq))
    assert torch.equal(few[0], all_[0][:40]) and torch.equal(few[2], all_[2][:, :40])
    assert torch.equal(few[1].view(torch.int32), all_[1][:40].view(torch.int32))
    ids, d = few[0].cpu().numpy(), few[1].cpu().numpy()
    finite = [i for i in range(40) if i != 5]
    assert (ids[finite, 0] != 3).all() and np.isfinite(d[finite, 0]).all()
    assert int(few[2][0, 5]) == 1  # one hop


@pytest.mark.parametrize("D", [32, 160])
@pytest.mark.parametrize("R", [16, 64])
def test_reverse_prune(vann_mod, D, R):
    """Inserts into a graph marked consistent (reverse re-prunes by the kernel that merges
    into lists in order) and into the same graph unmarked (every list sorted again): the
    same lists, with NaN rows among the old and the new, and FP32 sums that round."""
    import torch

    n, m = 1200, 260
    rng = np.random.default_rng(9)
    base = workload.mixture(n + m, D, 12, seed=405) * np.float32(1.0009765625)
    bad = rng.permutation(n + m)[:120]
    base[bad, 2] = np.nan
    entry = int(np.setdiff1d(np.arange(n), bad)[0])
    rows = torch.from_numpy(base).cuda()
    built = vann_mod.Index(D, R, 70, 1.2, capacity=n)
    built.build(rows[:n], batch=0, seed=3, entry=entry)
    _, deg, adj = built.get_graph()
    got = []
    for consistent in (True, False):
        idx = vann_mod.Index(D, R, 70, 1.2, capacity=n + m)
        idx.set_graph(base[:n], deg, adj, entry, consistent=consistent)
        idx.insert(rows[n:])
        got.append(idx.get_graph())
    (_, deg_a, adj_a), (_, deg_b, adj_b) = got
    assert np.array_equal(deg_a, deg_b)
    live = np.arange(R) < deg_a[:, None]
    assert np.array_equal(np.where(live, adj_a, 0), np.where(live, adj_b, 0))
    assert (adj_a[live] < n + m).all() and np.isin(adj_a[live], bad).any()
