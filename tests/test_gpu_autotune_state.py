"""The autotuner's trial steps leave the particles as they were: positions,
velocities, ids, and the last step's order, which restore_order still undoes."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 90000], ids=["small_step", "large_step"])
def test_autotune_leaves_ids_and_order(gpu, n):
    m = int(np.ceil(n ** (1 / 3)))
    sc = scenes.dam_break(m, m, m, (4.0, 4.0, 4.0), scene_id=331, n_keep=n)
    rng = np.random.default_rng(n)
    sc.x[:] = sc.x[rng.permutation(n)]
    sc.x[::50, 1] = 50.0  # outside the area: the step deletes them
    b = api.Batch(1, n, 300000, 30)
    i = b.add_scene(H.resolved(api.config_params(scorr_k=1e-4), sc), n, sc.domain_end, H.gpu_boundary(sc, "planes"),
                    sc.area, sc.x, sc.v)
    state = lambda: [*b.get_scene(i), b.particle_ids(i), *b.restore_order(i, n), *b.particles_by_id(i, n)]  # noqa: E731
    b.step(2)
    before = state()
    b.autotune(2)
    for k, (p, q) in enumerate(zip(before, state())):
        assert np.array_equal(p, q, equal_nan=p.dtype == np.float32), k
