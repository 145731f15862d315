"""The autotuner times the neighbour chunk only where the step depends on it:
with short lists (a batch whose scenes all expect at most 16 neighbours) and in
small steps the setting stays as it was, with large steps of long lists one of
the two is chosen.  The particles are left as they were."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [4, 8])
@pytest.mark.parametrize("n,long,kept", [(90000, False, True), (3000, True, True), (90000, True, False)],
                         ids=["short_lists", "small_step", "long_lists"])
def test_chunk_is_tuned_where_it_counts(gpu, n, long, kept, chunk):
    m = int(np.ceil(n ** (1 / 3)))
    sc = scenes.dam_break(m, m, m, (4.0, 4.0, 4.0), scene_id=330, n_keep=n)
    p = H.resolved(api.config_params(scorr_k=1e-4) if long else H.reflike_params(), sc)
    b = api.Batch(1, n, 300000, 30)
    i = b.add_scene(p, n, sc.domain_end, H.gpu_boundary(sc, "planes"), sc.area, sc.x, sc.v)
    for _ in range(3):  # (timings: a setting that is chosen by chance changes within a few)
        b.set_chunk(chunk)
        b.autotune(2)
        got = b.launch_shape()["chunk"]
        assert got == chunk if kept else got in (4, 8)
    x, v = b.get_scene(i)
    assert np.array_equal(x, sc.x) and np.array_equal(v, sc.v)
