"""The smallest steps' one-launch sort (prediction to reorder in a cluster)
against the kernel per phase that a profiled step launches: permutation, cell
ranges, lists, ids, positions and velocities bit for bit, for table sizes of
1, 2 and 4 rounds a block, particle counts up to the largest, deletions, and
buckets beyond a particle's own count (65, 300 and 5,000 members)."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _params(grid):
    return dict(api.config_params(scorr_k=1e-4), smoothing_length=0.1, cell_width=0.1, grid_size=list(grid))


def _positions(n, grid, pile, gone, seed):
    g = np.random.default_rng(seed)
    x = (g.random((n, 3)) * np.asarray(grid) * 0.1).astype(np.float32)
    for k, m in enumerate(pile):  # m particles of one cell, spread over the input order
        at = g.permutation(n)[:m]
        x[at] = np.float32(0.1 * (2 + k)) + g.random((len(at), 3)).astype(np.float32) * np.float32(0.05)
    x[g.permutation(n)[:gone], 1] = 60.0
    return x, g.normal(scale=0.1, size=(n, 3)).astype(np.float32)


@pytest.mark.parametrize("n,grid,pile,gone", [
    (1, (4, 4, 4), (), 0), (33, (2, 2, 2), (), 0), (255, (8, 8, 8), (65,), 1), (4096, (16, 16, 16), (64, 300), 100),
    (6000, (32, 32, 16), (5000,), 0), (10001, (32, 32, 32), (), 70), (16384, (32, 32, 32), (66, 66), 0),
    (16000, (64, 32, 16), (), 16000)])
def test_front_equals_a_kernel_per_phase(gpu, n, grid, pile, gone):
    x, v = _positions(n, grid, pile, gone, n)
    p = _params(grid)
    area = ((-1e3, -1.0, -1e3), (1e3, 50.0, 1e3))
    out = []
    for profiled in (False, True):
        part = api.PbfParticle(p, n, np.asarray(grid, np.float32) * 0.1)
        part.set_particles(x, v)
        for _ in range(2):
            if profiled:
                assert "k_rank_reorder" in [k for k, _ in api.profile_step(part, None, area, 2)]
            else:
                api.one_step(part, None, area, 2)
        d = part.neighbor_debug()
        xo, vo = part.get_particles()
        out.append([d[k] for k in ("sorted_hash", "perm", "cell_start", "cell_end", "neighbor_list")] +
                   [xo.view(np.uint32), vo.view(np.uint32), part.particle_ids(), np.array([d["num"], part.flags()]),
                    np.array([part.launches])])
    assert out[0].pop()[0] == out[1].pop()[0] - 5  # one launch in place of six
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), k


def test_front_packed_scenes_equal_a_kernel_per_phase(gpu):
    import torch
    sizes = [(700, (8, 8, 8), (65,), 3), (1, (4, 4, 4), (), 0), (3000, (16, 16, 8), (), 0), (0, (8, 8, 8), (), 0)]
    rows = [_positions(n, g, p, d, 50 + k) if n else (np.zeros((0, 3), np.float32),) * 2
            for k, (n, g, p, d) in enumerate(sizes)]
    counts = np.array([r[0].shape[0] for r in rows], np.uint32)
    x, v = (torch.tensor(np.concatenate([r[k] for r in rows]), device="cuda") for k in (0, 1))
    out = []
    for packed in (True, False):
        b = api.Batch(4, 16384, 16384, 30)
        ids = [b.add_scene(_params(g), 4096, np.asarray(g, np.float32) * 0.1, None,
                           ((-1e3, -1.0, -1e3), (1e3, 50.0, 1e3)), np.full((1, 3), 0.15, np.float32), None)
               for _, g, _, _ in sizes]
        if packed:
            b.step_packed(2, x, v, counts)
        else:
            b.set_all(x, v, counts)
            b.profile_step(2)
        out.append([a.view(np.uint32) for i in ids for a in b.get_scene(i)])
    for k, (a, c) in enumerate(zip(*out)):
        assert np.array_equal(a, c), k
