"""The blur with taps that run the other way (a negative radius, or a negative
scale): the order of a pixel's taps is reversed, so the texels past either
border are other taps'.  Against the oracle's blur, whose taps are all clamped.

Tolerance: two expf a weight, within 3 ulp of the oracle's each, a product and
a sum: a pixel's normalised weights agree to 2 x 8 x 2^-23 = 1.9e-6, the
linear depths they average lie within 1, and a depth changes by at most 4
times the linear depth at the nearest particles (l > 0.03): 1e-5."""
import numpy as np
import pytest

from oracle import ssf as S
from ssf_pbf_cuda_gb300 import api
from tests.test_gpu_ssf_tiles import _cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,scale", [(-5.5e-6, 1.0), (-2e-4, 1.0), (-0.05, 1.0), (2e-4, -1.0), (-2e-4, -1.0)],
                         ids=["inside", "edges", "outside", "scale", "both"])
@pytest.mark.parametrize("size", [(129, 66), (5, 3), (1, 1)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_blur_with_reversed_taps(gpu, size, radius, scale):
    p = api.ssf_default_params(width=size[0], height=size[1], blur_passes=1, point_radius=1.5, blur_radius=radius)
    p["blur_scale"] *= scale
    r = api.SsfRenderer(p)
    r.render(_cloud(r, 3000, 9, "mixed"))
    inv, inc = r.frame_constants()
    got, want = r.image("blurred"), S.blur(S.frame(r.params, inv, inc), r.image("blur_input"))
    assert np.array_equal(got == 1, want == 1)
    assert np.max(np.abs(got - want)) <= 1e-5
