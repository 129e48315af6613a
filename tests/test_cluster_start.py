"""A kernel that reaches into the shared memory of the other blocks of its
cluster passes a cluster barrier first: only then have they all started (the
sources are read; no GPU needed)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "flecsph_gb300", "csrc")


def test_cluster_barrier_before_first_remote_access():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for kernel in re.split(r"(?=__global__)", src)[1:]:
            remote = kernel.find("map_shared_rank")
            if remote < 0:
                continue
            seen += 1
            before = kernel[:remote]
            arrive = before.find(".barrier_arrive()")
            assert ".sync()" in before or 0 <= arrive < before.find(".barrier_wait()"), path
    assert seen
