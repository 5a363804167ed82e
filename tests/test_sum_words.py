"""A long sum's search words (SumWords) are clear before and after every sum: the
kernel that ends the sum clears them, and where a launch fails on the way
(out of memory for a kernel's code, say) the host does.  Otherwise the next
difference would start from the failed one's top limb and could take the
smaller operand for the larger."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hypergeometrica_gb300", "csrc")


def test_failed_sum_clears_its_words():
    text = open(os.path.join(CSRC, "hg_crt.cu")).read()
    body = re.search(r"cudaError_t launch_large_sum\(.*?\n}", text, re.S).group(0)
    last = body.index("launch_dep(sum_finish_kernel")
    failed = re.search(r"if \(e != cudaSuccess\) \{(.*?)\n  \}", body[last:], re.S)
    assert failed, "no clean-up after the last launch"
    assert "cudaMemsetAsync(words, 0xff, 2 * sizeof(long long), st)" in failed.group(1)
    assert "cudaMemsetAsync(&words->done, 0" in failed.group(1)
    struct = re.search(r"struct SumWords \{(.*?)\};", open(os.path.join(CSRC, "hg_internal.h")).read(), re.S).group(1)
    assert re.findall(r"(?:long long|unsigned) (\w+);", struct) == ["top_diff", "top_out", "done"]
