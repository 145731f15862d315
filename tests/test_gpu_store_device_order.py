"""A copy to device arrays returns when the stream has come to it: pinned
memory that the stream wrote before holds its data then, with no further
wait, as when the call waited for the stream itself."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu


def test_pinned_memory_written_before_the_copy_is_there(gpu):
    import torch
    sc = scenes.dam_break(10, 10, 10, (2.0, 2.0, 2.0), scene_id=321)
    part = api.PbfParticle(H.resolved(api.config_params(scorr_k=1e-4), sc), sc.n, sc.domain_end)
    stream = torch.cuda.Stream()
    src = torch.zeros(1 << 18, dtype=torch.int32, device="cuda")
    dst = torch.zeros(1 << 18, dtype=torch.int32).pin_memory()
    view = dst.numpy()
    x, v = torch.zeros((sc.n, 3), device="cuda"), torch.zeros((sc.n, 3), device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        part.set_particles(sc.x, sc.v, stream)
        for k in range(1, 41):
            src.fill_(k)
            dst.copy_(src, non_blocking=True)
            part.get_particles_device(x, v, stream)
            assert (view == k).all()
    stream.synchronize()
    assert np.array_equal(x.cpu().numpy(), sc.x)
