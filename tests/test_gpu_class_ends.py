"""Alias-class ranges at the edges of their 8-bit ends: buckets of two classes
whose member counts straddle the sizes at which the rank kernels change (16,
64) and the class bytes end (254 members grouped by class, 255 walked whole),
in the small steps' rank and the large steps'.  Lists equal the oracle's slot
for slot."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _scene(sizes, filler: int) -> scenes.Scene:
    """Buckets of a 16^3 table of 0.1 m cells holding sizes[k] particles, one in
    four of them in the cell 16 cells along x (the same bucket, another class);
    filler particles spread over other cells."""
    rng = np.random.default_rng(5)
    parts = []
    for k, m in enumerate(sizes):
        cell = np.array([1 + 2 * (k % 6), 2 + 3 * (k // 6), 4], np.float64)
        x = (cell + rng.uniform(0.05, 0.95, size=(m, 3))) * 0.1
        x[::4, 0] += 1.6
        parts.append(x)
    parts.append(np.stack([rng.uniform(0.0, 3.2, filler), rng.uniform(0.0, 1.6, filler), rng.uniform(0.8, 1.6, filler)], 1))
    x = np.concatenate(parts).astype(np.float32)
    x = x[rng.permutation(len(x))]
    return scenes.Scene(x, np.zeros_like(x), (3.2, 1.6, 1.6), ((-0.2,) * 3, (3.4, 1.8, 1.8)),
                        scenes.box_planes((3.2, 1.6, 1.6)), (16, 16, 16))


@pytest.mark.parametrize("filler", [500, 140000], ids=["small_step", "large_step"])
def test_class_ranges_at_bucket_size_edges(oracle, gpu, filler):
    sc = _scene([1, 2, 15, 16, 17, 63, 64, 65, 253, 254, 255, 256, 300], filler)
    params = api.config_params(scorr_k=1e-4, body_force=[0.0, 0.0, 0.0])
    g = H.run_gpu(sc, params, "planes", iters=0)
    r = H.run_oracle(oracle, sc, params, "planes", iters=0)
    H.assert_integer_parity(g, r, H.resolved(params, sc))
