"""Small steps' wide list reads at list lengths around their batches (16 and
32 slots) and rows, u16 and u32 lists, several scenes a tile list: positions
and velocities equal the large steps' passes bit for bit (the same scenes in a
batch with enough filler to be a large step)."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _scenes():
    # spacing from h / 2 (33 neighbours within h) to beyond h (none)
    out = []
    for k, (n, sp) in enumerate([(63, 0.05), (64, 0.06), (257, 0.045), (1000, 0.0375), (300, 0.12), (1, 0.05)]):
        m = int(np.ceil(n ** (1 / 3)))
        out.append(scenes.dam_break(m, m, m, (2.0, 2.0, 2.0), scene_id=300 + k, spacing=sp, n_keep=n,
                                    origin=(0.3, 0.3, 0.3)))
    return out


def _run(scs, params, filler, max_pair, capacity, steps=4):
    small = [(sc, H.resolved(params, sc)) for sc in scs]
    side = {False: 0, True: 52, "mid": 32}[filler]
    fill = [scenes.dam_break(side, side, side, (4.0, 4.0, 4.0), scene_id=390)] if side else []
    rest = [(sc, H.resolved(params, sc)) for sc in fill]
    cells = sum(int(np.prod(p["grid_size"])) + 1 for _, p in small + rest)
    b = api.Batch(len(small) + len(rest), sum(max(sc.n, capacity) for sc, _ in small + rest), cells, max_pair)
    ids = []
    for sc, p in small + rest:
        bnd = api.Boundary(points_on_planes=sc.planes[0], normals_on_planes=sc.planes[1])
        ids.append(b.add_scene(p, max(sc.n, capacity), sc.domain_end, bnd, sc.area, sc.x, sc.v))
    b.step(steps)
    return [b.get_scene(i) for i in ids[:len(small)]]


@pytest.mark.parametrize("capacity", [0, 70000], ids=["u16", "u32"])
@pytest.mark.parametrize("max_pair", [9, 17, 30, 34, 70])
def test_small_step_lists_equal_large_steps(gpu, max_pair, capacity):
    params = api.config_params(scorr_k=1e-4, max_pair_particle_num=max_pair)
    scs = _scenes()[:3] if capacity else _scenes()
    small = _run(scs, params, False, max_pair, capacity)
    large = _run(scs, params, True, max_pair, capacity)
    for k, ((xa, va), (xb, vb)) in enumerate(zip(small, large)):
        assert len(xa) == scs[k].n
        assert np.array_equal(xa.view(np.uint32), xb.view(np.uint32)), k
        assert np.array_equal(va.view(np.uint32), vb.view(np.uint32)), k


@pytest.mark.parametrize("capacity", [0, 70000], ids=["u16", "u32"])
@pytest.mark.parametrize("max_pair", [9, 16, 18, 30, 34, 70])
def test_lanes_and_one_lane_lists_equal(gpu, max_pair, capacity):
    """Two lanes a particle (few particles) against one (32,768 more): sums
    pass from lane to lane in list order."""
    params = api.config_params(scorr_k=1e-4, max_pair_particle_num=max_pair)
    scs = _scenes()[:3] if capacity else _scenes()
    for k, ((xa, va), (xb, vb)) in enumerate(zip(_run(scs, params, False, max_pair, capacity),
                                                 _run(scs, params, "mid", max_pair, capacity))):
        assert np.array_equal(xa.view(np.uint32), xb.view(np.uint32)), k
        assert np.array_equal(va.view(np.uint32), vb.view(np.uint32)), k


@pytest.mark.parametrize("filler", [False, "mid", True], ids=["small", "mid", "large"])
@pytest.mark.parametrize("capacity", [0, 70000], ids=["u16", "u32"])
def test_infinite_velocities_count_listed_neighbours_only(gpu, capacity, filler):
    """Pairs far apart from each other whose confinement overflows to opposite
    infinite velocities: XSPH adds c (v_j - v_i) W for the one listed neighbour
    (the particle itself is not listed), inf - inf = NaN in every component;
    the slots past a list's end, whose loads are the particle's own, add
    nothing (their v_i - v_i = NaN would trip the pass's NaN guard)."""
    params = api.config_params(scorr_k=1e-4, vc_parameter=float("inf"))
    rng = np.random.default_rng(5)
    m = 5
    c = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.3 + 0.3
    off = rng.normal(size=c.shape)
    off *= 0.03 / np.linalg.norm(off, axis=1, keepdims=True)
    sc = scenes.dam_break(m, m, 2 * m, (2.0, 2.0, 2.0), scene_id=310, spacing=0.05)
    sc.x = np.concatenate([c + off, c - off]).astype(np.float32)
    sc.v = rng.normal(scale=0.1, size=sc.x.shape).astype(np.float32)
    xs, vs = _run([sc], params, filler, params["max_pair_particle_num"], capacity, steps=1)[0]
    assert len(xs) == sc.n and np.isfinite(xs).all()
    assert np.isnan(vs).all()
