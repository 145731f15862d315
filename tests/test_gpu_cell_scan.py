"""The cell-count scan at the table sizes where its form changes: one block of
registers, a cluster of blocks, three kernels (tables are the grid's cells and
one deleted bucket).  Cell ranges and permutation equal the oracle's."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 1), (8, 8, 16), (16, 16, 16), (32, 16, 16), (32, 32, 16), (32, 32, 32), (64, 32, 32), (64, 64, 32),
         (64, 64, 64), (128, 64, 64)]


@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
def test_cell_ranges_by_table_size(oracle, gpu, grid):
    rng = np.random.default_rng(17)
    box = tuple(0.1 * g for g in grid)
    x = (rng.uniform(-0.05, 1.05, size=(9001, 3)) * box).astype(np.float32)  # some outside the area: deleted
    sc = scenes.Scene(x, np.zeros_like(x), box, ((0.0,) * 3, box), scenes.box_planes(box), grid)
    params = api.config_params(scorr_k=1e-4, body_force=[0.0, 0.0, 0.0])
    for graph in (True, False):
        g = H.run_gpu(sc, params, "planes", iters=0, steps=1, graph=graph)
        r = H.run_oracle(oracle, sc, params, "planes", iters=0)
        H.assert_integer_parity(g, r, H.resolved(params, sc))
