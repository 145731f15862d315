"""The depth splat by pixel tiles (particle sets beyond the box raster's bound)
and by pixel boxes at that bound: image sides that are no multiple of a tile,
sprites from one pixel to the whole image, particles clipped at every border,
near-to-far and far-to-near order.  The depth image is bit-exact against the
oracle's splat."""
import numpy as np
import pytest

from oracle import ssf as S
from ssf_pbf_cuda_gb300 import api

pytestmark = pytest.mark.gpu


def _cloud(r, n, seed, order):
    """n particles around the camera, none within its sphere of the eye plane
    (the splat's early rejection supposes a front point before the eye)."""
    g = np.random.default_rng(seed)
    x = (g.uniform(-1, 1, (2 * n, 3)) * np.array([14, 10, 30]) + np.array([2, 4, -5])).astype(np.float32)
    v = np.asarray(r.params["view"], np.float64).reshape(4, 4)
    ez = x @ v[:3, 2] + v[3, 2]
    x = x[(ez < -r.params["point_radius"] - 0.2) | (ez > r.params["point_radius"])][:n]
    assert len(x) == n
    k = np.argsort(x[:, 2], kind="stable")
    return x[k if order == "far_first" else k[::-1]] if order != "mixed" else x


@pytest.mark.parametrize("n", [19999, 20000, 20001, 40000])
@pytest.mark.parametrize("size", [(333, 197), (64, 36), (7, 3), (1, 1)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_depth_by_tiles_is_exact(gpu, n, size):
    for order in ("mixed", "near_first", "far_first"):
        r = api.SsfRenderer(api.ssf_default_params(width=size[0], height=size[1], blur_passes=0))
        x = _cloud(r, n, n + size[0], order)
        for _ in range(2):  # the tile bounds start afresh on every frame
            r.render(x)
            inv, inc = r.frame_constants()
            assert np.array_equal(r.image("depth"), S.splat(S.frame(r.params, inv, inc), x)), order


@pytest.mark.parametrize("radius", [0.002, 0.18, 6.0], ids=["points", "default", "huge"])
@pytest.mark.parametrize("mode", [api.L.PBF_SSF_SPLAT_QUAD, api.L.PBF_SSF_SPLAT_SPRITE])
def test_depth_by_tiles_at_sprite_sizes(gpu, mode, radius):
    r = api.SsfRenderer(api.ssf_default_params(width=101, height=67, blur_passes=1, splat_mode=mode, point_radius=radius))
    x = _cloud(r, 25000, 3, "mixed")
    r.render(x)
    inv, inc = r.frame_constants()
    assert np.array_equal(r.image("depth"), S.splat(S.frame(r.params, inv, inc), x))


@pytest.mark.parametrize("radius", [5.5e-6, 2e-4, 0.05], ids=["inside", "edges", "outside"])
@pytest.mark.parametrize("size", [(129, 66), (5, 3), (1, 1)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_blur_taps_inside_and_past_the_edges(gpu, size, radius):
    """Taps within a texel, at the borders' texels and past every border,
    against the oracle's blur (expf differs by a few ulps: 2e-6, as the other
    passes' tests allow)."""
    r = api.SsfRenderer(api.ssf_default_params(width=size[0], height=size[1], blur_passes=1, point_radius=1.5,
                                               blur_radius=radius))
    r.render(_cloud(r, 3000, 9, "mixed"))
    inv, inc = r.frame_constants()
    got, want = r.image("blurred"), S.blur(S.frame(r.params, inv, inc), r.image("blur_input"))
    assert np.array_equal(got == 1, want == 1)
    assert np.max(np.abs(got - want)) <= 2e-6
