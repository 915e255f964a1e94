"""Several host threads, an index each: the same kernels launched at different sizes at
the same time."""
import threading

import numpy as np
import pytest

from vann import workload

pytestmark = pytest.mark.gpu


def _together(work):
    """Runs the callables at once; their exceptions, if any."""
    start, errors = threading.Barrier(len(work)), []

    def go(f):
        start.wait()
        try:
            f()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=go, args=(f,)) for f in work]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return errors


@pytest.mark.parametrize("store", ["f32", "bf16"])
@pytest.mark.parametrize("D,Ls", [(128, (64, 32)), (128, (100, 70)), (128, (256, 130)), (128, (512, 300)),
                                  (192, (1000, 400)), (384, (128, 66))])
def test_searches_of_different_sizes(vann_mod, D, Ls, store):
    import torch

    base = torch.from_numpy(workload.mixture(1500, D, 12, seed=421)).cuda()
    q = base[:4].contiguous()
    work, outs, want = [], [], []
    for L in Ls:
        idx = vann_mod.Index(D, 32, 40, 1.2, capacity=1500, stores=("f32", "bf16"))
        idx.build(base, batch=0, seed=5)
        out = (torch.empty((4, 5), dtype=torch.int32, device="cuda"), torch.empty((4, 5), device="cuda"))
        outs.append(out)
        stream = torch.cuda.Stream()

        def go(idx=idx, L=L, out=out, stream=stream):
            for i in range(4000):
                idx.search(q, k=5, L=L, store=store, out=out, stream=stream)
                if i % 256 == 255:
                    stream.synchronize()
            stream.synchronize()

        work.append(go)
    torch.cuda.synchronize()
    assert _together(work) == []
    for f, out in zip(work, outs):
        idx, L = f.__defaults__[:2]
        ids, d = idx.search(q, k=5, L=L, store=store)
        assert torch.equal(ids, out[0]) and torch.equal(d, out[1])


def test_builds_of_different_widths(vann_mod):
    """Prunes ask for shared memory by row length and candidate count."""
    import torch

    work, graphs = [], [[], []]
    for t, (D, R, L) in enumerate(((64, 32, 60), (128, 64, 90))):
        base = torch.from_numpy(workload.mixture(1500, D, 12, seed=422)).cuda()

        def go(D=D, R=R, L=L, base=base, got=graphs[t]):
            stream = torch.cuda.Stream()
            for stores in (("f32", "u8"), ("f32",)) * 3:
                idx = vann_mod.Index(D, R, L, 1.2, capacity=1500, stores=stores)
                idx.build(base, batch=500, seed=5, stream=stream)
                _, deg, adj = idx.get_graph()
                got.append(np.where(np.arange(R) < deg[:, None], adj, -1))
                idx.close()

        work.append(go)
    torch.cuda.synchronize()
    assert _together(work) == []
    for got in graphs:
        assert all(np.array_equal(got[0], g) for g in got)
