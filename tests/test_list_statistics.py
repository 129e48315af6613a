"""The walk keeps the list statistics up to the size at which the pair passes
stop asking for them: one number in the sources (no GPU needed)."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "flecsph_gb300", "csrc")


def test_one_limit():
    def text(name):
        return open(os.path.join(CSRC, name)).read()
    assert re.search(r"#define SPLIT_MAX LIST_STAT_MAX", text("fsph_mixed_kernels.cuh"))
    assert re.search(r"P\.n <= LIST_STAT_MAX", text("fsph_tree.cu"))
    assert len(re.findall(r"P\.n <= SPLIT_MAX", text("fsph_mixed.cu"))) == 3
