"""Particles copied to device arrays before the host knows their count: the
live particles only, in the order and bits of the host copy, the entries past
them untouched, at block edges of the copy, after deletions and when none is
left."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [False, True], ids=["default_stream", "side_stream"])
@pytest.mark.parametrize("n,gone", [(1, 0), (1, 1), (255, 3), (256, 0), (257, 1), (1000, 1000), (3000, 1700)])
def test_device_copy_counts_on_the_device(gpu, n, gone, side):
    import torch
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    m = int(np.ceil(n ** (1 / 3)))
    sc = scenes.dam_break(m, m, m, (2.0, 2.0, 2.0), scene_id=320, n_keep=n)
    p = H.resolved(api.config_params(scorr_k=1e-4), sc)
    x = np.array(sc.x, np.float32)
    x[n - gone:, 1] = 50.0  # outside the area: the step deletes them
    part = api.PbfParticle(p, n, sc.domain_end)
    bnd = H.gpu_boundary(sc, "planes")
    with torch.cuda.stream(stream):
        part.set_particles(x, sc.v, stream)
        xo, vo = (torch.full((n, 3), 7.0, device="cuda") for _ in range(2))
        stream.synchronize()
        for _ in range(2):  # the second copy's bound is the count
            api.one_step(part, bnd, sc.area, 4, stream)
            part.get_particles_device(xo, vo, stream)
            stream.synchronize()
            xh, vh = part.get_particles(stream)
            assert len(xh) == n - gone
            for dev, host in ((xo, xh), (vo, vh)):
                got = dev.cpu().numpy()
                assert np.array_equal(got[:n - gone].view(np.uint32), host.view(np.uint32))
                assert (got[n - gone:] == 7.0).all()
