"""Orders that the CUDA sources must keep and that no run is sure to show
broken, read from the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ssf_pbf_cuda_gb300", "csrc")


def _source(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)


def _body(src, at):
    """The braced block that follows position at."""
    start = src.index("{", at)
    depth = 0
    for k in range(start, len(src)):
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        if depth == 0:
            return src[start:k + 1]
    raise AssertionError("unbalanced braces")


def test_cluster_scan_meets_before_it_writes_other_blocks():
    src = _source("pbf_scan.cuh")
    body = _body(src, src.index("cluster_scan("))
    arrive, wait, write = (body.find(k) for k in ("barrier.cluster.arrive", "barrier.cluster.wait", "map_shared_rank"))
    assert 0 <= arrive < wait < write
    # callers that skip the barrier have met before
    for name in ("pbf_kernels.cu", "pbf_noalloc.cu"):
        src = _source(name)
        for m in re.finditer(r"cluster_scan<R, true>", src):
            kernel = src[src.rindex("__global__", 0, m.start()):m.start()]
            assert "cluster.sync()" in kernel or "barrier_wait" in kernel
