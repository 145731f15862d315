"""Calls whose kernels are set up while the one before runs, where a missing
dependency would show: many calls with different inputs enqueued one after the
other without a wait, and calls recorded in a graph and replayed on other
inputs.  Sorts against a stable sort by cell, frames against frames rendered
alone."""
import ctypes

import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api
from ssf_pbf_cuda_gb300._lib import check

pytestmark = pytest.mark.gpu


class _Sort:
    def __init__(self, n, grid, device):
        import torch
        self.grid, self.cells = grid, int(np.prod(grid))
        self.x = torch.zeros((n, 3), device=device)
        self.out = [torch.full((m,), -5, dtype=torch.int32, device=device) for m in (max(n, 1), self.cells, self.cells)]

    def enqueue(self, stream):
        n = self.x.shape[0]
        check(api.load().pbf_cell_sort_noalloc(self.x.data_ptr(), n, 0.25, (ctypes.c_uint32 * 3)(*self.grid),
                                               *[t.data_ptr() for t in self.out], stream.cuda_stream), "sort")

    def check(self):
        x = self.x.cpu().numpy()
        c = np.floor(x / np.float32(0.25)).astype(np.int64) % np.array(self.grid)
        key = (c[:, 2] * self.grid[1] + c[:, 1]) * self.grid[0] + c[:, 0]
        want = np.argsort(key, kind="stable")
        b = np.searchsorted(key[want], np.arange(self.cells + 1))
        none = b[1:] == b[:-1]
        perm, start, end = (t.cpu().numpy().view(np.uint32) for t in self.out)
        assert np.array_equal(perm[:len(x)], want.astype(np.uint32))
        assert np.array_equal(start, np.where(none, 0xFFFFFFFF, b[:-1]).astype(np.uint32))
        assert np.array_equal(end, np.where(none, 0xFFFFFFFF, b[1:]).astype(np.uint32))


def _points(n, grid, seed, pile=0):
    import torch
    g = np.random.default_rng(seed)
    x = g.uniform(0.0, 1.0, size=(n, 3)) * np.array(grid) * 0.25
    x[:pile] = 0.1
    return torch.from_numpy(x[g.permutation(n)].astype(np.float32))


# (particles, table, piled in one cell): each form of the scan and of the rank
SORTS = [(3000, (8, 8, 8), 0), (0, (32, 32, 32), 0), (30000, (4, 4, 4), 0), (100000, (32, 32, 32), 9000),
         (5000, (128, 64, 64), 2000), (1, (4, 4, 4), 0), (262144, (64, 64, 64), 0), (70000, (16, 16, 16), 30000)]


def test_sorts_enqueued_without_a_wait(gpu):
    import torch
    stream = torch.cuda.Stream()
    sorts = [_Sort(n, grid, gpu) for n, grid, _ in SORTS * 3]
    for k, (s, (n, grid, pile)) in enumerate(zip(sorts, SORTS * 3)):
        s.x.copy_(_points(n, grid, k, pile))
    torch.cuda.synchronize()
    for s in sorts:
        s.enqueue(stream)
    stream.synchronize()
    for s in sorts:
        s.check()


@pytest.mark.parametrize("n,grid,pile", SORTS, ids=[f"{n}" for n, _, _ in SORTS])
def test_recorded_sorts_replay_on_other_inputs(gpu, n, grid, pile):
    import torch
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    a, b = _Sort(n, grid, gpu), _Sort(n, grid, gpu)
    a.enqueue(stream)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        a.enqueue(stream)
        b.enqueue(stream)
    for k in range(3):
        for j, s in enumerate((a, b)):
            s.x.copy_(_points(n, grid, 10 * k + j, pile))
        torch.cuda.synchronize()
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        a.check()
        b.check()


# (particles, width, height, blur passes): both rasters, one and eight row blocks
FRAMES = [(32768, 320, 180, 3), (500, 64, 36, 3), (0, 333, 197, 1), (25000, 333, 197, 0), (60000, 640, 360, 3),
          (3000, 1600, 1000, 2)]


def _cloud(n, seed):
    g = np.random.default_rng(seed)
    return (g.uniform(-1, 1, (n, 3)) * [4, 3, 6] + [2, 2, -2]).astype(np.float32)


def _renderer(w, h, blurs):
    return api.SsfRenderer(api.ssf_default_params(width=w, height=h, blur_passes=blurs))


def _images(r):
    return [r.image(k) for k in ("depth", "blurred", "normal", "color", "rgba8")]


def _same(a, b):
    assert all(np.array_equal(p, q, equal_nan=True) for p, q in zip(a, b))


def test_frames_enqueued_without_a_wait(gpu):
    import torch
    stream = torch.cuda.Stream()
    sets = [(f, torch.from_numpy(_cloud(f[0], k)).cuda()) for k, f in enumerate(FRAMES * 2)]
    renderers = [_renderer(*f[1:]) for f, _ in sets]
    torch.cuda.synchronize()
    for _ in range(2):  # (each renderer's frame before is of another set)
        for r, (f, x) in zip(renderers, sets[1:] + sets[:1]):
            r.render(x, stream)
        for r, (f, x) in zip(renderers, sets):
            r.render(x, stream)
    stream.synchronize()
    for r, (f, x) in zip(renderers, sets):
        alone = _renderer(*f[1:])
        alone.render(x)
        _same(_images(r), _images(alone))


@pytest.mark.parametrize("frame", FRAMES, ids=[f"{n}_{w}x{h}" for n, w, h, _ in FRAMES])
def test_recorded_frames_replay_on_other_inputs(gpu, frame):
    import torch
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    r, other = _renderer(*frame[1:]), _renderer(*frame[1:])
    x = torch.from_numpy(_cloud(frame[0], 1)).cuda()
    for q in (r, other):
        q.render(x, stream)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        r.render(x, stream)
        other.render(x, stream)
    for k in range(3):
        x.copy_(torch.from_numpy(_cloud(frame[0], 20 + k)))
        torch.cuda.synchronize()
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        alone = _renderer(*frame[1:])
        alone.render(x)
        for q in (r, other):
            _same(_images(q), _images(alone))
