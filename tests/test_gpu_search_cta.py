"""Small batches run a CTA per query (search_cta.cuh), large ones a warp per query: the same
queries must give the same ids, distances and work counts either way, at the edges of the
worklist, list and row sizes each takes."""
import numpy as np
import pytest

from vann import workload

pytestmark = pytest.mark.gpu

BIG = 1200  # queries: more than 7 per SM on 148 SMs, so the warp kernels take the batch


def _index(vann_mod, n, D, R, stores, integer=True, seed=201):
    import torch

    base = workload.mixture(n, D, 12, seed=seed, sigma=20.0 if integer else 0.05, integer=integer, unit_norm=not integer)
    idx = vann_mod.Index(D, R, 48, 1.2, capacity=n + 64, stores=stores)
    idx.build(torch.from_numpy(base).cuda(), batch=0, seed=5)
    q = workload.mixture(BIG, D, 12, seed=seed + 1, sigma=20.0 if integer else 0.05, integer=integer, unit_norm=not integer)
    return idx, q


def _same(idx, q, small, **kw):
    import torch

    qd = torch.from_numpy(q).cuda()
    few = idx.search_stats(qd[:small].contiguous(), **kw)
    all_ = idx.search_stats(qd, **kw)
    assert torch.equal(few[0], all_[0][:small]) and torch.equal(few[1], all_[1][:small])
    assert torch.equal(few[2], all_[2][:, :small])


@pytest.mark.parametrize("D,R,store,integer", [(16, 32, "u8", True), (48, 20, "u8", True), (128, 64, "u8", True),
                                               (144, 64, "u8", True), (512, 96, "u8", True), (4, 64, "f32", True),
                                               (100, 33, "f32", False), (128, 128, "f32", True), (384, 64, "f32", False),
                                               (96, 64, "bf16", False), (256, 64, "bf16", False), (128, 64, "fp8", True),
                                               (272, 40, "fp8", False)])
@pytest.mark.parametrize("L,k", [(1, 1), (32, 10), (64, 64), (65, 10), (128, 100), (129, 10), (256, 256)])
def test_small_batch_equals_large(vann_mod, D, R, store, integer, L, k):
    idx, q = _index(vann_mod, 1500, D, R, ("f32", store) if store != "f32" else ("f32",), integer)
    for kw in ({}, {"quirks": 1, "rerank": True}, {"max_hops": 3}):
        _same(idx, q, 37, k=k, L=L, store=store, **kw)


def test_tombstones_uneven_and_one_query(vann_mod):
    import torch

    idx, q = _index(vann_mod, 2000, 128, 64, ("f32", "u8"))
    entry = idx.info()["entry"]
    idx.delete(torch.tensor([entry] + list(range(0, 400, 3)), dtype=torch.int32, device="cuda"))
    for L in (48, 100):
        _same(idx, q, 1, k=10, L=L, store="u8")
        _same(idx, q, 300, k=L, L=L, store="f32")
    qd = torch.from_numpy(q).cuda()
    rng = np.random.default_rng(3)
    L = torch.from_numpy(rng.integers(1, 121, BIG).astype(np.int32)).cuda()
    k = torch.minimum(L, torch.from_numpy(rng.integers(1, 31, BIG).astype(np.int32)).cuda())
    L[0], k[0] = 120, 30
    few = idx.search_uneven(qd[:50].contiguous(), L[:50].contiguous(), k[:50].contiguous(), store="u8")
    all_ = idx.search_uneven(qd, L, k, store="u8")
    assert torch.equal(few[0], all_[0][:50]) and torch.equal(few[1], all_[1][:50])


@pytest.mark.parametrize("L", [32, 100])
def test_distances_that_overflow_end_the_search(vann_mod, L):
    """A query whose squared distances are +inf: no candidate is closer than anything."""
    idx, q = _index(vann_mod, 600, 128, 32, ("f32",))
    q[:3] = 3e38
    q[3, 5] = 2e19
    _same(idx, q, 20, k=10, L=L)


def test_small_inserts_equal_the_oracle(oracle, vann_mod):
    """Insert searches of a few rows run a CTA per row: expansion lists and all, one batch
    after the other (snapshot filter, R = 64, L over the register sizes)."""
    import torch

    n0, R, L = 1200, 64, 130
    base = workload.mixture(n0 + 60, 128, 12, seed=211)
    for stores in (("f32",), ("f32", "u8")):
        og, entry = oracle.build_index(base[:n0], R=R, L=L, alpha=1.2, seed=5, skip_mode=2,
                                       bloom_mode=oracle.BLOOM_SNAPSHOT)
        deg, adj = np.zeros(n0 + 60, np.uint32), np.zeros((n0 + 60, R), np.uint32)
        deg[:n0], adj[:n0] = og.deg, og.adj
        g = oracle.Graph(base, deg, adj)
        idx = vann_mod.Index(128, R, L, 1.2, capacity=n0 + 60, stores=stores)
        idx.build(torch.from_numpy(base[:n0]).cuda(), batch=0, seed=5)
        at = n0
        for c in (1, 7, 52):
            idx.insert(torch.from_numpy(base[at:at + c]).cuda())
            assert g.vamana_batch(at, c, L, 1.2, entry, skip_mode=0, bloom_mode=oracle.BLOOM_SNAPSHOT) == 0
            at += c
        _, gdeg, gadj = idx.get_graph()
        assert all(np.array_equal(gadj[i, :gdeg[i]], g.adj[i, :g.deg[i]]) for i in range(n0 + 60))


def test_autotuning_on_a_small_batch_makes_no_choice(vann_mod):
    """A batch for the CTA-per-query kernel has one launch variant: one time for all, where
    a fastest of seven equal runs would be the choice of every later large batch."""
    import torch

    idx, q = _index(vann_mod, 1500, 128, 32, ("f32", "u8"))
    qd = torch.from_numpy(q).cuda()
    for store in ("f32", "u8"):
        ms = idx.autotune(qd[:64].contiguous(), k=10, L=48, store=store)
        assert len(set(ms)) == 1 and ms[0] > 0
    with pytest.raises(vann_mod.VannError):
        idx.autotune(qd, k=10, L=5)  # k > L
