"""Which search kernel and launch variant a batch gets (csrc/search_rule.h), on the CPU:
the edges of the rule, and the shapes where a variant other than 6 blocks per SM measured
slower than 6."""
import os
import subprocess

import pytest

from conftest import PKG

SMS = 148
F32, BF16, FP8, U8, PQ = range(5)
SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "search_rule.h"
int main() {
    unsigned long long nq; unsigned D, R, L, beam, iq; int store;
    const int blocks[] = {6, 4, 5, 7, 8, 9, 10};
    while (scanf("%llu %u %u %u %u %d %u", &nq, &D, &R, &L, &beam, &store, &iq) == 7) {
        const vann::SearchShape s{nq, D, R, L, beam, store, iq != 0};
        printf("%d %d\n", (int)vann::cta_per_query(s, 148), blocks[vann::search_variant(s, 148)]);
    }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(d / "t.cpp"), "-o", str(d / "t")], check=True)

    def ask(shapes):
        text = "\n".join(" ".join(str(int(v)) for v in s) for s in shapes)
        out = subprocess.run([str(d / "t")], input=text, check=True, capture_output=True, text=True).stdout
        return [tuple(int(v) for v in ln.split()) for ln in out.split("\n")[:-1]]

    return ask


def _s(nq, store=U8, L=64, R=64, D=128, beam=1, iq=False):
    return nq, D, R, L, beam, store, iq


def test_cta_per_query_edges(rule):
    for L, R, D, per in ((64, 64, 128, 4), (65, 64, 128, 7), (128, 64, 128, 7), (64, 65, 128, 7), (64, 64, 144, 7),
                         (129, 64, 128, 3), (256, 128, 512, 3), (257, 64, 128, 0)):
        for store in (F32, BF16, FP8, U8):
            got = rule([_s(max(1, per * SMS), store, L, R, D), _s(per * SMS + 1, store, L, R, D)])
            assert [g[0] for g in got] == [int(per > 0), 0], (L, R, D, store)
    assert [g[0] for g in rule([_s(1, PQ), _s(1, beam=2)])] == [0, 0]


@pytest.mark.parametrize("shape", [
    # two parents per hop: 8 blocks 2 to 9% slower than 6
    _s(10_000, L=32, beam=2), _s(10_000, L=64, beam=2), _s(5_000, L=32, beam=2),
    # long lists: 7 blocks up to 15% slower
    _s(10_000, L=300), _s(10_000, F32, L=300), _s(20_000, L=500), _s(10_000, L=300, iq=True), _s(10_000, L=200), _s(5_000, L=200)])
def test_no_more_blocks_than_measured(rule, shape):
    beam2 = shape[4] == 2
    assert rule([shape])[0][1] <= (7 if beam2 else 6)


@pytest.mark.parametrize("store,L", [(U8, 64), (U8, 200), (F32, 64), (F32, 300), (BF16, 100)])
def test_every_query_resident_where_they_fit(rule, store, L):
    """Up to 24 queries per SM none waits for a second round (blocks of 4 queries)."""
    for nq in (16 * SMS, 16 * SMS + 1, 20 * SMS, 20 * SMS + 1, 24 * SMS):
        assert rule([_s(nq, store, L)])[0][1] == -(-nq // (4 * SMS))


def test_shapes_with_one_variant(rule):
    got = rule([_s(nq, st, L, R, D) for nq in (2_000, 10_000) for st in (F32, U8) for L in (32, 300)
                for R, D in ((65, 128), (64, 132))] + [_s(10_000, PQ)])
    assert {g[1] for g in got} == {6}
