"""Every kernel that is launched through chain() waits for the kernel before it
in its first statement (the sources are read; no GPU needed)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "flecsph_gb300", "csrc")


def test_chained_kernels_wait_first():
    src = "".join(open(f).read() for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))))
    first = {}
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(", src):
        body = src.index("{", src.index(")", m.end()))
        first[m.group(1)] = src[body + 1:].lstrip().startswith("chain_begin();")
    chained = set()
    for pat in (r"chain\(L, (k_\w+)", r"DISPATCH\w*\((?:\w+, )?(k_\w+)",
                r"(k_\w+)<D, KK", r"cudaLaunchKernelEx\(&cfg, (k_\w+)"):
        found = set(re.findall(pat, src))
        assert found, pat
        chained |= found
    assert len(chained) > 25
    assert sorted(k for k in chained if not first[k]) == []
