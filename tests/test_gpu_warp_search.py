"""The warp-per-query kernels against the oracle: batches too large for a CTA per query, of
sizes that reach the launch variants of 4 to 8 blocks per SM (csrc/search_rule.h)."""
import numpy as np
import pytest

from vann import workload

pytestmark = pytest.mark.gpu


def _sizes():
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return [7 * sms + 64, 16 * sms + 51, 20 * sms + 50, 36 * sms + 77]


@pytest.fixture(scope="module")
def graphs(oracle):
    out = {}
    for R in (32, 64):
        base = workload.mixture(3000, 128, 40, seed=440 + R)
        out[R] = (base, *oracle.build_index(base, R=R, L=64, alpha=1.2, seed=3))
    return out


def _index(vann_mod, base, g, entry, stores):
    idx = vann_mod.Index(128, g.R, 64, 1.2, capacity=len(base), stores=stores)
    idx.set_graph(base, g.deg, g.adj, entry, consistent=True)
    return idx


@pytest.mark.parametrize("R,L,k,quirk", [(64, 10, 10, 0), (64, 64, 64, 1), (64, 150, 100, 0), (64, 300, 20, 1),
                                         (32, 32, 10, 1), (32, 75, 75, 0)])
def test_every_format_matches_the_oracle(oracle, vann_mod, graphs, R, L, k, quirk):
    """Integer rows and queries are exact in FP32, BF16 and uint8."""
    import torch

    base, g, entry = graphs[R]
    sizes = _sizes()
    q = workload.mixture(sizes[-1], 128, 40, seed=441)
    st, oids, od, _, _ = g.search(q, L, k, entry, skip_mode=quirk, bloom_mode=oracle.BLOOM_SNAPSHOT)
    assert st == 0
    idx = _index(vann_mod, base, g, entry, ("f32", "bf16", "u8"))
    qd = torch.from_numpy(q).cuda()
    for nq in sizes:
        for store in ("f32", "bf16", "u8"):
            ids, d = idx.search(qd[:nq].contiguous(), k=k, L=L, store=store, quirks=quirk)
            assert np.array_equal(ids.cpu().numpy().view(np.uint32), oids[:nq]), (nq, store)
            assert np.array_equal(d.cpu().numpy(), od[:nq]), (nq, store)


@pytest.mark.parametrize("L", [48, 100])
def test_autotuned_on_a_large_batch_is_exact(oracle, vann_mod, graphs, L):
    import torch

    base, g, entry = graphs[64]
    nq = _sizes()[0]
    q = workload.mixture(nq, 128, 40, seed=442)
    idx = _index(vann_mod, base, g, entry, ("f32", "u8"))
    qd = torch.from_numpy(q).cuda()
    _, oids, od, _, _ = g.search(q, L, 10, entry, bloom_mode=oracle.BLOOM_SNAPSHOT)
    for store in ("f32", "u8"):
        ms = idx.autotune(qd, k=10, L=L, store=store)
        assert len(ms) == vann_mod.lib().vann_search_variant_count() and min(ms) > 0
        ids, d = idx.search(qd, k=10, L=L, store=store)
        assert np.array_equal(ids.cpu().numpy().view(np.uint32), oids)
        assert np.array_equal(d.cpu().numpy(), od)


@pytest.mark.parametrize("R,L", [(64, 64), (64, 130), (32, 20)])
def test_fractional_queries_over_uint8_rows(vann_mod, graphs, R, L):
    """Queries that are not integers take the FP32 path over the uint8 rows, in the CTA and
    in the warp kernels alike; nearly the FP32 rows' results (another order of the sums)."""
    import torch

    base, g, entry = graphs[R]
    nq = _sizes()[1]
    q = workload.mixture(nq, 128, 40, seed=443) + np.float32(0.3)
    idx = _index(vann_mod, base, g, entry, ("f32", "u8"))
    qd = torch.from_numpy(q).cuda()
    few, all_ = (idx.search_stats(qd[:c].contiguous(), k=10, L=L, store="u8") for c in (300, nq))
    assert torch.equal(few[0], all_[0][:300]) and torch.equal(few[1], all_[1][:300])
    assert torch.equal(few[2], all_[2][:, :300])
    ids, d = idx.search(qd, k=10, L=L)
    same = ids == all_[0]
    assert float(same.float().mean()) > 0.99
    assert torch.allclose(d[same], all_[1][same], rtol=1e-5)


def test_uneven_large_batch(oracle, vann_mod, graphs):
    import torch

    base, g, entry = graphs[64]
    nq = _sizes()[0]
    q = workload.mixture(nq, 128, 40, seed=444)
    rng = np.random.default_rng(2)
    Ls = rng.choice([16, 40, 100, 180], nq).astype(np.int32)
    ks = np.minimum(Ls, rng.choice([1, 10, 50], nq)).astype(np.int32)
    idx = _index(vann_mod, base, g, entry, ("f32", "u8"))
    for store in ("f32", "u8"):
        ids, d = idx.search_uneven(torch.from_numpy(q).cuda(), torch.from_numpy(Ls).cuda(), torch.from_numpy(ks).cuda(),
                                   store=store)
        gi, gd = ids.cpu().numpy().view(np.uint32), d.cpu().numpy()
        for L in np.unique(Ls):
            rows = np.nonzero(Ls == L)[0]
            _, oids, od, _, _ = g.search(q[rows], int(L), int(L), entry, bloom_mode=oracle.BLOOM_SNAPSHOT)
            for r, oi, dd in zip(rows, oids, od):
                k = ks[r]
                assert np.array_equal(gi[r, :k], oi[:k]) and np.array_equal(gd[r, :k], dd[:k])
                assert (gi[r, k:] == 0xFFFFFFFF).all() and np.isinf(gd[r, k:]).all()
