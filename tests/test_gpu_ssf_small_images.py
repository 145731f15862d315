"""The splat's two rasters on both sides of the image sizes and particle counts
between which they are chosen, clouds before the camera and close to it: the
depth image is bit-exact against the oracle's splat."""
import numpy as np
import pytest

from oracle import ssf as S
from ssf_pbf_cuda_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("near", [False, True], ids=["before", "near"])
@pytest.mark.parametrize("size,n", [((128, 128), 20500), ((127, 130), 20500), ((192, 128), 30000), ((191, 129), 30000),
                                    ((192, 128), 262144), ((192, 128), 262145)], ids=str)
def test_depth_by_either_raster(gpu, size, n, near):
    r = api.SsfRenderer(api.ssf_default_params(width=size[0], height=size[1], blur_passes=0, point_radius=0.05))
    g = np.random.default_rng(n + size[0])
    x = g.uniform(-1, 1, (n, 3)) * ([1, 1, 1] if near else [6, 4, 12]) + ([2, 3, 8] if near else [2, 2, -4])
    x = x.astype(np.float32)
    for _ in range(2):
        r.render(x)
        inv, inc = r.frame_constants()
        assert np.array_equal(r.image("depth"), S.splat(S.frame(r.params, inv, inc), x))
