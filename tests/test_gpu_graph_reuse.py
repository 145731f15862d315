"""A batch whose scene set changes between steps: sets taken in turn, on either
side of the sizes and neighbour counts at which the launch shape changes, are
stepped by graphs captured once each, with the results of a fresh batch.  Each
case runs in a process of its own, whose runtime calls the profiler counts."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

# (particles, long lists): two lanes or one, small or large step, short or long
# lists, three sets in turn
CASES = {"lanes": [(24000, True), (25000, True)], "small_large": [(70000, True), (80000, True)],
         "lists": [(9000, True), (9000, False)], "lanes_short": [(9600, False), (9900, False)],
         "three": [(500, True), (30000, True), (90000, False)]}


@pytest.mark.parametrize("case", CASES)
def test_sets_in_turn_are_captured_once_each(gpu, case):
    r = subprocess.run([sys.executable, "-m", "tests.test_gpu_graph_reuse", case], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    launched, captured = (int(t) for t in r.stdout.split()[-2:])
    if launched == 0:
        pytest.skip("the profiler recorded no runtime calls")
    assert launched == 3 * len(CASES[case]) and captured == 0


def main(case):
    import torch
    from torch.profiler import ProfilerActivity, profile

    from ssf_pbf_cuda_gb300 import api, scenes
    from tests import helpers as H
    torch.cuda.init()
    params = {True: api.config_params(scorr_k=1e-4), False: H.reflike_params()}

    def add(b, n, long):
        m = int(np.ceil(n ** (1 / 3)))
        sc = scenes.dam_break(m, m, m, (4.0, 4.0, 4.0), scene_id=n, n_keep=n)
        p = H.resolved(params[long], sc)
        return b.add_scene(p, n, sc.domain_end, H.gpu_boundary(sc, "planes"), sc.area, sc.x, sc.v)

    def stepped(b, k):
        i = add(b, *CASES[case][k])
        b.step(2)
        x, v = b.get_scene(i)
        b.remove_scene(i)
        return x, v

    def same(p, q):
        assert all(np.array_equal(a.view(np.uint32), c.view(np.uint32)) for a, c in zip(p, q))

    turn = range(len(CASES[case]))
    fresh = [stepped(api.Batch(1, CASES[case][k][0], 300000, 30), k) for k in turn]
    b = api.Batch(2, 200000, 600000, 30)
    for k in turn:
        same(stepped(b, k), fresh[k])
    for _ in range(2):  # (the first profile of a process may miss calls)
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
            torch.zeros(1, device="cuda")
            for k in list(turn) * 3:
                same(stepped(b, k), fresh[k])
            torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    print(sum("GraphLaunch" in n for n in names), sum("GraphInstantiate" in n for n in names))


if __name__ == "__main__":
    main(sys.argv[1])
