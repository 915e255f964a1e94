"""The two sides of the CTA-per-query search meet at named barriers: __syncthreads is only
defined where all threads reach the same one, and the sides run different code."""
import os
import re

from conftest import PKG


def test_no_syncthreads_where_the_warps_part():
    text = open(os.path.join(PKG, "csrc", "search_cta.cuh")).read()
    sides = text[text.index("        if (warp == 0) {\n"):text.index("        n = ctl[1];")]
    worklist, gather = sides.split("        } else {\n            Query<S, DC> qv;")
    gather = gather[:gather.rindex("        }\n")]  # the barrier after the sides is common
    for side in (worklist, gather):
        assert "__syncthreads" not in side
        assert len(re.findall(r"hop_barrier\(\);", side)) == 2
