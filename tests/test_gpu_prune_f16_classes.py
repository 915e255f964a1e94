"""The float-row prune's passes for 128 and 256 candidates against a plain restatement with
the kernels' order of FP32 sums, over rows whose differences do not fit f16; rows with NaN
and infinite distances; an exact uint8 index whose row length the integer passes do not take."""
import numpy as np
import pytest

from test_gpu_prune_f16 import _dist_f32, _rows_equal
from vann import workload

pytestmark = pytest.mark.gpu


def _consolidated(vann_mod, base, R, alpha, hit, dead, seed):
    """Lists of `hit` nodes, which point at one or three of the `dead`, before and after
    consolidation."""
    import torch

    n, live = len(base), len(base) - len(dead)
    rng = np.random.default_rng(seed)
    deg = np.full(n, R, np.uint32)
    adj = np.stack([rng.permutation(live)[:R] for _ in range(n)]).astype(np.uint32)
    for i, p in enumerate(hit):
        for j, x in enumerate(dead if i % 3 == 0 else dead[:1]):
            adj[p, (7 * p + 5 * j) % R] = x
    idx = vann_mod.Index(base.shape[1], R, 64, float(alpha), capacity=n)
    idx.set_graph(base, deg, adj, entry=100)
    idx.delete(torch.tensor(dead, dtype=torch.int32, device="cuda"))
    idx.consolidate()
    _, gdeg, gadj = idx.get_graph()
    return adj, gdeg, gadj


def _expect(base, adj, p, dead, R, alpha):
    cand = []
    for x in adj[p]:
        cand += [int(x)] if x not in dead else [int(u) for u in adj[x]]
    cand = [c for c in dict.fromkeys(cand) if c != p and c not in dead]
    with np.errstate(over="ignore", invalid="ignore"):
        d = _dist_f32(base[p:p + 1], base[cand])[0]
        order = np.argsort(d.view(np.uint32) & 0x7FFFFFFF, kind="stable")  # a NaN last
        cand, d = np.array(cand)[order], d[order]
        pair = _dist_f32(base[cand], base[cand])
        live, chosen = np.ones(len(cand), bool), []
        for t in range(len(cand)):
            if live[t] and len(chosen) < R:
                chosen.append(cand[t])
                live &= ~(pair[t] * alpha <= d)
    return len(cand), chosen


# per SM: up to 4 nodes start at the 256-candidate pass, more at the 128-candidate one
@pytest.mark.parametrize("per_sm", [2, 6])
@pytest.mark.parametrize("D,alpha", [(60, 1.0), (60, 1.2), (128, 1.2)])
def test_decisions_in_every_pass(vann_mod, per_sm, D, alpha):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    R, hits, alpha = 60, per_sm * sms, np.float32(alpha)
    n = 2 * hits + 300
    rng = np.random.default_rng(D + per_sm)
    base = rng.integers(-4000, 4001, (n, D)).astype(np.float32)
    dead = [n - 3, n - 2, n - 1]
    hit = list(range(hits))
    adj, gdeg, gadj = _consolidated(vann_mod, base, R, alpha, hit, dead, seed=per_sm)
    sizes = []
    for p in hit[:: 4 if per_sm == 2 else 11]:  # a third of them have three deleted neighbours
        size, chosen = _expect(base, adj, p, dead, R, alpha)
        sizes.append(size)
        assert gadj[p, :gdeg[p]].tolist() == chosen, p
    assert min(sizes) <= 128 < max(sizes) <= 256


@pytest.mark.parametrize("per_sm", [2, 6])
def test_nan_and_infinite_rows(vann_mod, per_sm):
    """A candidate at +inf leaves every test of its node to FP32, a NaN one prunes nothing
    and is pruned by nothing."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    R, D, hits, alpha = 60, 64, per_sm * sms, np.float32(1.2)
    n = 2 * hits + 300
    rng = np.random.default_rng(31)
    base = rng.integers(-4000, 4001, (n, D)).astype(np.float32)
    odd = rng.permutation(n - 3)[: n // 40]
    base[odd[::2], 3] = np.nan
    base[odd[1::2], 5] = 3e38
    dead = [n - 3, n - 2, n - 1]
    hit = [p for p in range(hits)]
    adj, gdeg, gadj = _consolidated(vann_mod, base, R, alpha, hit, dead, seed=9)
    for p in hit[::max(1, hits // 60)] + [int(o) for o in odd if o < hits][:8]:
        _, chosen = _expect(base, adj, p, dead, R, alpha)
        assert gadj[p, :gdeg[p]].tolist() == chosen, p


@pytest.mark.parametrize("D", [16, 48, 112])
def test_exact_bytes_of_odd_length(oracle, vann_mod, D):
    """Row lengths of 16 but not 32: uint8 distances from the search, f16 passes in the prune."""
    import torch

    n, m, R = 1700, 90, 32
    base = workload.mixture(n + m, D, 15, seed=451)
    og, entry = oracle.build_index(base[:n], R=R, L=75, alpha=1.2, seed=7, skip_mode=2, bloom_mode=oracle.BLOOM_SNAPSHOT)
    rows, got = torch.from_numpy(base).cuda(), []
    for stores in (("f32", "u8"), ("f32",)):
        idx = vann_mod.Index(D, R, 75, 1.2, capacity=n + m, stores=stores)
        idx.build(rows[:n], batch=0, seed=7)
        _, deg, adj = idx.get_graph()
        assert idx.info()["entry"] == entry and idx.info()["pruned_tc"] == 0
        assert _rows_equal(deg, adj, og.deg, og.adj) == []
        for at in range(n, n + m, 30):
            idx.insert(rows[at: at + 30])
        got.append(idx.get_graph())
    assert _rows_equal(got[0][1], got[0][2], got[1][1], got[1][2]) == []
