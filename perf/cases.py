"""The engine's work as its users give it, one case per way of using it.

``listed()`` names them, ``draw()`` gives more of the same ranges, ``prepare()`` makes
what a program holds before the call (rows, queries, a built index), ``run()`` is one
pass through the public entry points, ``work()`` the bytes and operations a pass cannot
do without and ``exact()`` the FP64 value of the distances it returns.

Kinds:

* ``search``: one batch of queries over a built index (``Index.search``).  Every row
  format the traversal has, with and without the exact rerank.
* ``build``: an index built from rows on the device (``Index.build``) and its lists
  fetched for the program's own use (``vann_get_graph`` into pinned host memory).
* ``live``: a few rows arrive and a few queries follow them (``Index.insert``, then
  ``Index.search``): the online mix of a serving process.
* ``churn``: a share of the index is deleted, consolidated away and replaced, then
  queried (``delete``, ``consolidate``, ``insert``, ``search``).
* ``loop``: one round of the reference driver's loop through its class (``Vamana``):
  insertPoints, deletePoints by vector, searchPoints2, patchGraph.

Rows are of the two kinds the engine is configured for: ``bytes``, integer-valued FP32
in [0, 255] from a clipped mixture (the shape of SIFT descriptors; the uint8 copy is then
exact), and ``unit``, a mixture around unit vectors (the shape of learnt embeddings; the
uint8 copy is then scalar quantization).
"""
from __future__ import annotations

import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cs5013-project_b200"))
import vann  # noqa: E402

ALPHA = 1.2
FIRST_BATCH = 10_000  # rows per build batch, as the 1M benchmark builds
POOL_PASSES = 40_000  # a live index keeps room for this many passes' rows


def listed() -> list:
    return [
        # one user's request on an idle server: the latency of a single query
        search("one query, bytes", "bytes", 1_000_000, 128, 64, "u8", False, 1, 64, 10),
        # what a server admits at once under light load: tens of queries on float rows
        search("small batch, unit rows", "unit", 200_000, 96, 64, "f32", False, 50, 100, 10),
        # the 1M x 128 benchmark's batch on the uint8 copy at its operating point
        search("benchmark batch, bytes", "bytes", 1_000_000, 128, 64, "u8", False, 10_000, 32, 10),
        # the reference's compile-time search configuration: 10,000 records, whole worklist of 199
        search("reference search, L=199", "bytes", 10_000, 128, 64, "f32", False, 10_000, 199, 199),
        # the reduced-precision configuration: float rows from the fitted uint8 grid, exact rerank
        search("quantized rerank, unit rows", "unit", 1_000_000, 96, 64, "u8", True, 10_000, 64, 10),
        # wide embeddings in BF16 with many results asked for, a mid-sized batch
        search("wide bf16 rerank", "unit", 100_000, 256, 64, "bf16", True, 1_000, 128, 100),
        # FP8 traversal at the benchmark's FP8 operating point, an odd batch size
        search("fp8 rerank, bytes", "bytes", 300_000, 128, 64, "fp8", True, 2_999, 40, 10),
        # index construction on byte rows, in the benchmark's batches
        build("build, bytes", "bytes", 300_000, 128, 64, "u8", 100, FIRST_BATCH),
        # index construction on float rows (every prune on FP32 rows), ragged last batch
        build("build, unit rows", "unit", 100_001, 96, 64, "f32", 100, FIRST_BATCH),
        # the online mix: ten rows arrive, ten queries follow
        live("live insert and search", "bytes", 1_000_000, 128, 64, "u8", 10, 10, 64, 10),
        # a FreshVamana round: 5% deleted and replaced, then queried at the churn benchmark's L
        churn("churn of 5%", "bytes", 300_000, 128, 64, "u8", 15_000, 1_000, 100, 10),
        # one round of the reference driver's workload loop over its class
        loop("reference class loop", "bytes", 20_000, 128, 64, 500, 1_000, 100),
    ]


def search(name, data, n, D, R, store, rerank, nq, L, k):
    return {"name": name, "kind": "search", "data": data, "n": n, "D": D, "R": R, "store": store, "rerank": rerank,
            "nq": nq, "L": L, "k": k}


def build(name, data, n, D, R, store, build_L, batch):
    return {"name": name, "kind": "build", "data": data, "n": n, "D": D, "R": R, "store": store, "build_L": build_L,
            "batch": batch}


def live(name, data, n, D, R, store, m, nq, L, k):
    return {"name": name, "kind": "live", "data": data, "n": n, "D": D, "R": R, "store": store, "m": m, "nq": nq,
            "L": L, "k": k}


def churn(name, data, n, D, R, store, m, nq, L, k):
    return {"name": name, "kind": "churn", "data": data, "n": n, "D": D, "R": R, "store": store, "m": m, "nq": nq,
            "L": L, "k": k}


def loop(name, data, n, D, R, m, nq, L):
    return {"name": name, "kind": "loop", "data": data, "n": n, "D": D, "R": R, "m": m, "nq": nq, "L": L}


def _log(rng, lo: int, hi: int) -> int:
    """A whole number spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng) -> dict:
    """One more case of the same ranges: searches half of the time, else updates and builds."""
    data = rng.choice(["bytes", "unit"])
    R = rng.choice([32, 48, 64, 64])
    kind = rng.choice(["search"] * 5 + ["build", "build", "live", "churn", "loop"])
    if kind == "search":
        D = rng.choice([64, 96, 128, 128, 192, 256])
        store, rerank = rng.choice([("f32", False), ("u8", data == "unit"), ("bf16", True), ("fp8", True)])
        n, nq, L = _log(rng, 10_000, 300_000), _log(rng, 1, 10_000), _log(rng, 16, 200)
        c = search("", data, n, D, R, store, rerank, nq, L, rng.choice([1, 10, min(100, L), L]))
        c["k"] = min(c["k"], L)
    elif kind == "build":
        D = rng.choice([64, 96, 128])
        n = _log(rng, 5_000, 100_000)
        c = build("", data, n, D, R, "u8" if data == "bytes" else "f32", rng.choice([64, 75, 100]),
                  rng.choice([FIRST_BATCH, 4_000, max(1_000, n // 5)]))
    elif kind == "live":
        c = live("", data, _log(rng, 20_000, 300_000), rng.choice([96, 128]), R, "u8" if data == "bytes" else "f32",
                 _log(rng, 1, 30), _log(rng, 1, 100), rng.choice([32, 64, 100]), 10)
    elif kind == "churn":
        n = _log(rng, 20_000, 200_000)
        c = churn("", data, n, rng.choice([96, 128]), R, "u8" if data == "bytes" else "f32",
                  int(n * rng.uniform(0.005, 0.05)), _log(rng, 10, 1_000), rng.choice([64, 100]), 10)
    else:
        n = _log(rng, 5_000, 20_000)
        c = loop("", data, n, 128, R, _log(rng, 50, 500), _log(rng, 10, 1_000), rng.choice([75, 100, 128]))
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs
def _rows(case: dict, count: int, gen: torch.Generator, centres: torch.Tensor) -> torch.Tensor:
    """``count`` rows of the case's mixture."""
    D = case["D"]
    lab = torch.randint(0, centres.shape[0], (count,), generator=gen, device="cuda")
    x = torch.randn((count, D), generator=gen, device="cuda")
    if case["data"] == "bytes":
        return x.mul_(20.0).add_(centres[lab]).round_().clamp_(0.0, 255.0).contiguous()
    return x.mul_(0.05).add_(centres[lab]).contiguous()


def _inputs(case: dict, seed: int) -> dict:
    """Rows and queries of a case, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, D = case["n"], case["D"]
    if case["data"] == "bytes":  # about a thousand rows per centre
        centres = torch.rand((max(20, n // 1000), D), generator=gen, device="cuda") * 255.0
    else:  # about five hundred rows per unit vector
        centres = torch.randn((max(20, n // 500), D), generator=gen, device="cuda")
        centres /= centres.norm(dim=1, keepdim=True)
    out = {"base": _rows(case, n, gen, centres)}
    if "nq" in case:
        out["queries"] = _rows(case, case["nq"], gen, centres)
    if case["kind"] == "live":
        out["pool"] = _rows(case, case["m"] * POOL_PASSES, gen, centres)
    elif case["kind"] in ("churn", "loop"):
        out["fresh"] = _rows(case, case["m"], gen, centres)
        out["gone"] = torch.randperm(n, generator=gen, device="cuda")[: case["m"]].to(torch.int32)
    return out


def _index(case: dict, capacity: int, build_L: int = 100) -> vann.Index:
    stores = ["f32", case["store"]] if case["store"] != "f32" else ["f32"]
    return vann.Index(case["D"], case["R"], build_L, ALPHA, capacity=capacity, stores=stores)


def prepare(case: dict, seed: int) -> dict:
    x = _inputs(case, seed)
    s = {"case": case, **x}
    n, m = case["n"], case.get("m", 0)
    if case["kind"] == "loop":
        s["index"] = vann.Vamana(x["base"], R=case["R"], L=case["L"], capacity=n + 4 * m, seed=7)
        s["gone"] = x["base"][x["gone"].long()].contiguous()
        return s
    if case["kind"] == "build":
        s["index"] = _index(case, n, case["build_L"])
        s["deg"] = torch.empty(n, dtype=torch.int32, pin_memory=True)
        s["adj"] = torch.empty((n, case["R"]), dtype=torch.int32, pin_memory=True)
        return s
    s["index"] = _index(case, n + m * (POOL_PASSES if case["kind"] == "live" else 1))
    s["index"].build(x["base"], batch=FIRST_BATCH, seed=7)
    s["at"] = 0
    return s


def _search(s: dict):
    c = s["case"]
    # byte rows are searched as they are; the fitted grid of float rows needs its rerank
    rerank = c.get("rerank", c["store"] == "u8" and c["data"] == "unit")
    return s["index"].search(s["queries"], k=c["k"], L=c["L"], store=c["store"], rerank=rerank)


def run(s: dict) -> dict:
    c, index = s["case"], s["index"]
    if c["kind"] == "search":
        ids, d = _search(s)
        return {"ids": ids, "dists": d}
    if c["kind"] == "build":
        index.build(s["base"], batch=c["batch"], seed=7)
        st = vann.lib().vann_get_graph(index._h, None, s["deg"].data_ptr(), s["adj"].data_ptr())
        if st != vann.OK:
            raise vann.VannError(st, vann.lib().vann_last_error().decode())
        # the lists go on to a program's own kernels, padded with -1 past each node's degree
        deg, adj = s["deg"].cuda(non_blocking=True), s["adj"].cuda(non_blocking=True)
        slot = torch.arange(c["R"], dtype=torch.int32, device="cuda")
        return {"deg": deg, "lists": adj.masked_fill_(slot >= deg[:, None], -1)}
    if c["kind"] == "live":
        rows = s["pool"][s["at"]: s["at"] + c["m"]]
        s["at"] = (s["at"] + c["m"]) % s["pool"].shape[0]
        new = index.insert(rows)
        ids, d = _search(s)
        return {"new": new, "ids": ids, "dists": d}
    if c["kind"] == "churn":
        index.delete(s["gone"])
        index.consolidate()
        s["gone"] = index.insert(s["fresh"])
        ids, d = _search(s)
        return {"new": s["gone"], "ids": ids, "dists": d}
    index.insertPoints(s["fresh"])
    index.deletePoints(s["gone"])
    rows = index.searchPoints2(s["queries"])
    index.patchGraph()
    s["fresh"], s["gone"] = s["gone"], s["fresh"]  # the next round brings back what this one took out
    return {"rows": rows}


# ---------------------------------------------------------------- what a pass cannot do without
_ROW_BYTES = {"f32": 4.0, "bf16": 2.0, "fp8": 1.0, "u8": 1.0}


def _search_work(n, D, R, L, nq, k, row_bytes, rerank):
    """A greedy search expands its whole worklist (a dozen more on the way to it) and
    measures about 22 new rows per expansion; a batch reads no list or row twice."""
    hops = L + 12
    rows = min(n, 22 * hops)
    read = min(nq * (hops * 4 * R + rows * row_bytes), n * (4 * R + row_bytes))
    if rerank:
        read += min(nq * L, n) * 4 * D
    return read + nq * (4 * D + 8 * k), nq * rows * 3 * D


def work(case: dict) -> dict:
    n, D, R, kind = case["n"], case["D"], case["R"], case["kind"]
    row = D * _ROW_BYTES[case.get("store", "f32")]
    if kind == "search":
        b, f = _search_work(n, D, R, case["L"], case["nq"], case["k"], row, case["rerank"])
        return {"bytes": b, "flops": f}

    def inserted(m, of, L):
        """Search and prune of m rows (a chosen neighbour is compared with the ~100
        candidates still open), and about one comparison list per reverse edge's target."""
        _, f = _search_work(of, D, R, L, m, 0, row, False)
        return m * (4 * D + 4 * R), f + m * R * 100 * 3 * D

    if kind == "build":
        b, f = inserted(n, n, case["build_L"])
        return {"bytes": b + n * 4 * (R + 1), "flops": f}
    m = case["m"]
    bi, fi = inserted(m, n, 100 if kind != "loop" else case["L"])
    bs, fs = _search_work(n, D, R, case["L"], case["nq"], case.get("k", case["L"]), row, False)
    b, f = bi + bs, fi + fs
    if kind in ("churn", "loop"):
        b += n * 4 * R  # every list is looked through for the deleted ids
        hit = min(n, m * R)  # lists that lost a neighbour are pruned again
        b += hit * 4 * R
        f += hit * R * 100 * 3 * D
    if kind == "loop":
        b += n * 4 * D + case["nq"] * case["L"] * 4 * D  # rows matched by value, rows returned
        f += case["nq"] * m * 3 * D  # queries against the insert list
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- FP64 values
def exact(case: dict, seed: int):
    """The k smallest FP64 squared distances of every query, for searches of the exact
    rows whose worklist is long enough for their index that they find these neighbours.
    Other searches are approximate by design (a query can miss its whole cluster), and
    ids, lists and returned rows have no such value."""
    if case["kind"] != "search" or case["store"] != "f32" or case["n"] > 12_000 or case["L"] < 128:
        return None
    x = _inputs(case, seed)
    base = x["base"].double()
    norms = base.square().sum(1)
    out = []
    for q in x["queries"].double().split(2_000):
        d = torch.addmm(norms, q, base.T, alpha=-2.0)
        d += q.square().sum(1, keepdim=True)
        out.append(d.topk(case["k"], dim=1, largest=False).values)
    return {"ids": None, "dists": torch.cat(out).clamp_(min=0.0)}
