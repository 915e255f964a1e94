"""The staged merge's tiles and slot classes: list lengths around a tile of 32 rows,
worklists at the edges of the register classes, short and long rows, duplicates, a row
output off 16-byte alignment; bit for bit against the oracle's merge."""
import ctypes as C

import numpy as np
import pytest

from vann import workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,L,n_stage,nq", [(4, 1, 1, 3), (100, 33, 31, 700), (128, 128, 32, 150), (128, 129, 33, 20),
                                            (64, 256, 65, 1300), (512, 257, 200, 9), (512, 1000, 40, 5), (128, 40, 0, 10)])
def test_merge_matches_oracle(oracle, vann_mod, D, L, n_stage, nq):
    import torch

    n = 700
    base = workload.mixture(n, D, 8, seed=301)
    il = workload.mixture(max(n_stage, 1), D, 8, seed=302)
    il[::3] = base[: len(il[::3])]  # equal distances: the earlier candidate stays
    il[1::7] = il[0]
    q = workload.mixture(nq, D, 8, seed=303)
    idx = vann_mod.Index(D, 32, 48, 1.2, capacity=n)
    idx.build(torch.from_numpy(base).cuda(), batch=0, seed=3)
    if n_stage:
        idx.stage_insert(torch.from_numpy(il).cuda())
    qd = torch.from_numpy(q).cuda()
    wids, _ = idx.search(qd, k=L, L=L)
    oids, od = oracle.merge_rerank(base, q, wids.cpu().numpy().view(np.uint32), il[:n_stage])
    ids, d, rows = idx.search_staged(qd, L=L, with_vecs=True)
    gi = ids.cpu().numpy().view(np.uint32)
    assert np.array_equal(gi, oids) and np.array_equal(d.cpu().numpy(), od)
    all_rows = np.concatenate([base, il[:n_stage], np.zeros((1, D), np.float32)])
    at = np.where(gi == 0xFFFFFFFF, len(all_rows) - 1, np.where(gi >= 0x80000000, n + (gi & 0x7FFFFFFF), gi))
    assert np.array_equal(rows.cpu().numpy(), all_rows[at])
    # the row output may start anywhere
    buf = torch.zeros(nq * L * D + 1, device="cuda")
    sp = vann_mod.SearchParams(L, L, 0, 0, 0, 0, 1)
    st = vann_mod.lib().vann_search_staged(idx._h, C.c_void_p(qd.data_ptr()), nq, C.byref(sp), C.c_void_p(ids.data_ptr()),
                                           C.c_void_p(d.data_ptr()), C.c_void_p(buf.data_ptr() + 4), None)
    torch.cuda.synchronize()
    assert st == 0 and torch.equal(buf[1:].view(nq, L, D), rows)
