"""The tensor-core prune's walk over its Gram tiles (csrc/gram_tiles.h), on the CPU: every
tile on and below the diagonal once and in order, and nothing issued or waited for after a
wait that gave up."""
import os
import subprocess

import pytest

from conftest import PKG

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "gram_tiles.h"
template <uint32_t COLS> void walk(uint32_t m, int fail) {
    int waits = 0;
    if (m > 0) printf("issue 0 0\n");
    const bool ok = vann::gram_tiles<COLS>(
        m, [&](uint32_t r) { printf("row %u\n", r); }, [&](uint32_t r, uint32_t c) { printf("issue %u %u\n", r, c); },
        [&]() { printf("wait\n"); return ++waits != fail; }, [&](uint32_t r, uint32_t c) { printf("read %u %u\n", r, c); },
        [&](bool late) { return late; });
    printf("%s\n", ok ? "ok" : "gave up");
}
int main(int, char** v) {
    const uint32_t m = atoi(v[2]);
    if (atoi(v[1]) == 64) walk<64>(m, atoi(v[3])); else walk<128>(m, atoi(v[3]));
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiles")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return lambda cols, m, fail: subprocess.run([str(d / "t"), str(cols), str(m), str(fail)], check=True,
                                                capture_output=True, text=True).stdout.split("\n")[:-1]


@pytest.mark.parametrize("cols,m", [(64, 0), (64, 1), (64, 64), (64, 65), (64, 128), (128, 128), (128, 129), (128, 256),
                                    (128, 576), (128, 768)])
def test_tiles_and_giving_up(walk, cols, m):
    tiles = [(r, c) for r in range((m + 127) // 128) for c in range(-(-min(m, 128 * (r + 1)) // cols))]
    lines = walk(cols, m, 0)
    assert [ln for ln in lines if ln.startswith("issue")] == [f"issue {r} {c}" for r, c in tiles]
    assert [ln for ln in lines if ln.startswith("read")] == [f"read {r} {c}" for r, c in tiles]
    assert lines[-1] == "ok" and lines.count("wait") == len(tiles)
    for fail in range(1, len(tiles) + 1):
        lines = walk(cols, m, fail)
        assert lines[-1] == "gave up"
        assert lines.count("wait") == fail and sum(ln.startswith("issue") for ln in lines) == fail
