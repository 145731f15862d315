"""Hash tables with an axis of one cell: the walk visits such an axis's cell
three times, so a particle meets itself (and its neighbours) more than once
and lists hold it again.  Large steps whose lists are collected in shared
memory and those whose lists are stored directly (max_pair from 98 on at a
tile of 256), u32 and u16 lists: slot for slot the oracle's, and the same bits
as small steps."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _sheet(grid, n, seed):
    """n particles over the table's cells, two deep along its axis of one cell
    (aliases of the same cell); 0.1 m cells."""
    g = np.random.default_rng(seed)
    box = np.asarray(grid) * 0.1
    box[np.asarray(grid) == 1] = 0.2
    x = (g.uniform(0.0, 1.0, size=(n, 3)) * box).astype(np.float32)
    b = tuple(float(t) for t in box + 0.1)
    return scenes.Scene(x, np.zeros_like(x), b, ((-0.5,) * 3, tuple(t + 0.5 for t in b)), scenes.box_planes(b),
                        tuple(grid))


def _params(max_pair):
    return api.config_params(scorr_k=1e-4, body_force=[0.0, 0.0, 0.0], max_pair_particle_num=max_pair)


@pytest.mark.parametrize("max_pair", [30, 97, 98, 256])
@pytest.mark.parametrize("grid", [(1, 64, 64), (64, 1, 32), (64, 64, 1), (1, 1, 4096)],
                         ids=lambda g: "x".join(map(str, g)))
def test_lists_of_large_steps(oracle, gpu, grid, max_pair):
    sc = _sheet(grid, 79000, max_pair)
    params = _params(max_pair)
    g = H.run_gpu(sc, params, "planes", iters=0)
    r = H.run_oracle(oracle, sc, params, "planes", iters=0)
    H.assert_integer_parity(g, r, H.resolved(params, sc))


@pytest.mark.parametrize("max_pair", [30, 98, 256])
@pytest.mark.parametrize("grid", [(1, 32, 32), (32, 32, 1)], ids=lambda g: "x".join(map(str, g)))
def test_u16_lists_of_large_steps_equal_small_ones(gpu, grid, max_pair):
    params = _params(max_pair)
    scs = [_sheet(grid, 27000, 7 * max_pair + k) for k in range(3)]
    out = []
    for group in (scs, scs[:1], scs[1:2], scs[2:]):  # one large step, three small ones
        cells = int(np.prod(grid)) + 1
        b = api.Batch(len(group), 27000 * len(group), cells * len(group), max_pair)
        ids = [b.add_scene(H.resolved(params, sc), sc.n, sc.domain_end, H.gpu_boundary(sc, "planes"), sc.area, sc.x, sc.v)
               for sc in group]
        b.step(2)
        out.append([a.view(np.uint32) for i in ids for a in b.get_scene(i)])
    for k, (a, c) in enumerate(zip(out[0], out[1] + out[2] + out[3])):
        assert np.array_equal(a, c), k
