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


def test_kernels_set_up_early_read_plainly_what_launches_before_them_write():
    """__ldg and const __restrict__ promise data that nobody writes while the
    kernel runs; a kernel that waits in after_previous runs while the launch
    before it writes.  The caller's own input may be read so."""
    inputs = {"x", "n_dev", "xp"}
    seen = 0
    for name in ("pbf_ssf.cu", "pbf_noalloc.cu"):
        src = _source(name)
        helpers = {m.group(1): m for m in re.finditer(r"__device__ [^;{}]*?\b(\w+)\(([^{};]*)\)\s*\{", src)}
        for m in re.finditer(r"__global__[^;{}]*?\b(\w+)\((?=[^()]*\b[A-Z]\w*\b|[^()]*\*)([^{};]*)\)\s*\{", src):
            body = _body(src, m.end() - 1)
            if "after_previous" not in body:
                continue
            seen += 1
            parts = [(m.group(2), body)]
            for h, hm in helpers.items():
                if re.search(r"\b%s\(" % h, body):
                    parts.append((hm.group(2), _body(src, hm.end() - 1)))
            for args, text in parts:
                for q in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", args):
                    assert q in inputs, (name, m.group(1), q)
                for q in re.findall(r"__ldg\(\s*(\w+)", text):
                    assert q in inputs, (name, m.group(1), q)
    assert seen >= 10  # set-up, two rasters, blur, normal, shade; scan, scatter, rank, big


def test_the_polled_count_is_a_release_read_by_acquire():
    engine, kernels = _source("pbf_engine.cu"), _source("pbf_kernels.cu")
    body = _body(engine, engine.index("Batch::store_device"))
    assert "volatile" not in body and "__atomic_load_n(slot, __ATOMIC_ACQUIRE)" in body
    assert not re.search(r"=\s*\*slot|\*slot\s*[!=]=", body)
    body = _body(kernels, kernels.index("void k_store_phase"))
    assert 0 <= body.find("fence.acq_rel.sys") < body.find("st.relaxed.sys")
