"""A step recorded in a caller's graph (graph mode off) and replayed after the
particle counts changed: the launches read the counts on the device, so a
replay is a step of whatever the batch then holds, with more tiles than at
capture too.  Against a batch that steps directly, bit for bit."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes

pytestmark = pytest.mark.gpu

AREA = ((-1e3, -1.0, -1e3), (1e3, 50.0, 1e3))


def _batch(n0, cap, grid, x, v, graph):
    p = dict(api.config_params(scorr_k=1e-4), grid_size=list(grid))
    b = api.Batch(2, 2 * cap, 2 * (int(np.prod(grid)) + 1), 30)
    b.set_graph_mode(graph)
    planes = scenes.box_planes((3.0, 3.0, 3.0))
    bnd = api.Boundary(points_on_planes=planes[0], normals_on_planes=planes[1])
    for _ in range(2):
        b.add_scene(p, cap, (3.0, 3.0, 3.0), bnd, AREA, x[:n0], v[:n0])
    return b


@pytest.mark.parametrize("grid", [(16, 16, 16), (32, 32, 32)], ids=["4k_cells", "32k_cells"])
@pytest.mark.parametrize("at,counts", [(700, [(1, 700), (1500, 700), (20000, 3), (30000, 30000)]),
                                       (20000, [(40, 60000), (60000, 60000), (300, 0)])],
                         ids=["from_700", "from_20000"])
def test_recorded_step_serves_later_counts(gpu, at, counts, grid):
    import torch
    cap = max(max(c) for c in counts)
    rng = np.random.default_rng(cap)
    m = int(np.ceil(cap ** (1 / 3)))
    x = scenes.lattice(m, m, m, 0.05, (0.15,) * 3)[:cap]
    x = torch.tensor((x + rng.uniform(-0.002, 0.002, size=x.shape)).astype(np.float32), device="cuda")
    v = torch.zeros_like(x)
    rec, ref = (_batch(at, cap, grid, x, v, graph) for graph in (False, True))
    xin, vin = torch.zeros((2 * cap, 3), device="cuda"), torch.zeros((2 * cap, 3), device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()

    def load(b, c):
        n = c[0] + c[1]
        xin[:n] = torch.cat([x[:c[0]], x[:c[1]]])
        b.set_all(xin[:n], vin[:n], np.array(c, np.uint32))
        b.live_counts()

    load(rec, (at, at))
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        rec.step(2, stream)
    for c in counts:
        for b, step in ((rec, graph.replay), (ref, lambda: ref.step(2))):
            load(b, c)
            torch.cuda.synchronize()
            step()
            torch.cuda.synchronize()
        (ca, xa, va), (cb, xb, vb) = rec.get_all(), ref.get_all()
        assert np.array_equal(ca, cb) and tuple(ca) == c
        assert np.array_equal(xa.view(np.uint32), xb.view(np.uint32))
        assert np.array_equal(va.view(np.uint32), vb.view(np.uint32))
