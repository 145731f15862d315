"""Frames on both sides of the image sizes between which the screen passes'
blocks are 8 rows high, with sides that are no multiple of a block: every pass
against the oracle's, as for the smaller frames."""
import pytest

from ssf_pbf_cuda_gb300 import api
from tests.test_gpu_ssf import _check_passes, _cloud, _frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1499, 1000), (1501, 1001), (2049, 1033), (4999, 2001)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_large_frame_pass_parity(gpu, size):
    r = api.SsfRenderer(api.ssf_default_params(width=size[0], height=size[1], blur_passes=2))
    x = _cloud(3000, 7)
    r.render(x)
    g = _check_passes(r, x, _frame(r))
    covered = g["depth"] < 1
    assert covered[-1, :].any() and covered[:, -1].any()
