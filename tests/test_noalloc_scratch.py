"""fsph_sort_keys_noalloc keeps its scratch between calls.  The one word of it
that its kernels read before they write it, the range's block counter, is set by
every call itself, so a call does not depend on how the one before it ended (the
source is read; no GPU needed)."""
import os
import re

TREE = os.path.join(os.path.dirname(__file__), "..", "flecsph_gb300", "csrc", "fsph_tree.cu")


def test_counter_cleared_before_the_range():
    src = re.sub(r"//[^\n]*", "", open(TREE).read())
    body = src[src.index("fsph_status fsph_sort_keys_noalloc("):]
    clear = re.search(r"cudaMemsetAsync\(range \+ RANGE_TICKET, 0, sizeof\(\*range\), L\.stream\)",
                      body)
    assert clear and clear.start() < body.index("launch_range(")
