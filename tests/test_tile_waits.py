"""A thread of the tensor-core prune whose wait gave up must not issue or wait for the
node's other tiles (up to 21, a second each).  No wait can be made to run out safely on a
GPU, so this reads the loop."""
import os
import re

from conftest import PKG


def test_giving_up_ends_issuing_and_waiting():
    text = open(os.path.join(PKG, "csrc", "prune_tc.cu")).read()
    loop = text[text.index("        bool late = false;"):text.index("if (__syncthreads_or(late))")]
    issues = re.findall(r"if \(([^\n]*)\) \{\n\s*tc_fence_after\(\);\n\s*issue_tile\(r, c\);", loop)
    assert issues == ["tid == 0 && !late"] and loop.count("issue_tile(") == 1
    # the phase moves with the waits, so that the last one issued can be waited for below
    waits = re.findall(r"if \(!late\) \{\n\s*late = !mbar_wait\(bar, phase\);\n\s*phase \^= 1u;\n\s*\}", loop)
    assert len(waits) == 1 and loop.count("mbar_wait(") == 1 and loop.count("phase ^= 1u") == 1
    after = text[text.index("if (__syncthreads_or(late))"):]
    assert "if (tid == 0 && late) mbar_wait(bar, phase ^ 1u);" in after[:300]
