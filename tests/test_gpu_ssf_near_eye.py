"""The splat's early rejection where a particle's front point is not its
nearest fragment: spheres that reach past the eye plane (their fragments lie at
any depth, down to 0), and a projection whose depth falls away from the eye.
Both rasters; the depth image is bit-exact against the oracle's."""
import numpy as np
import pytest

from oracle import ssf as S
from ssf_pbf_cuda_gb300 import api

pytestmark = pytest.mark.gpu


def _cloud(n, seed, spread):
    g = np.random.default_rng(seed)
    return (g.uniform(-1, 1, (n, 3)) * spread + np.array([2, 4, 10])).astype(np.float32)  # around the eye


@pytest.mark.parametrize("flip", [False, True], ids=["usual", "reversed_depth"])
@pytest.mark.parametrize("radius", [0.05, 0.3, 2.0])
@pytest.mark.parametrize("mode", [api.L.PBF_SSF_SPLAT_QUAD, api.L.PBF_SSF_SPLAT_SPRITE], ids=["quad", "sprite"])
@pytest.mark.parametrize("n", [3, 400, 21000])
def test_depth_around_the_eye_is_exact(gpu, n, mode, radius, flip):
    p = api.ssf_default_params(width=61, height=45, blur_passes=0, splat_mode=mode, point_radius=radius)
    if flip:
        p["projection"] = p["projection"].copy()
        p["projection"][[10, 14]] *= -1
    covered = 0
    for spread in (0.3, 1.0, 4.0):
        r = api.SsfRenderer(p)
        x = _cloud(n, n + int(10 * spread), spread)
        r.render(x)
        inv, inc = r.frame_constants()
        want = S.splat(S.frame(r.params, inv, inc), x)
        assert np.array_equal(r.image("depth"), want), spread
        covered += int((want < 1).sum())
    assert covered or n < 400
