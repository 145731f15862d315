"""Performance cases of the solver, the neighbour-search sort and the renderer.

Every case is one pass through the public entry points (`api.Batch`,
`api.PbfParticle`, `api.SsfRenderer`, `pbf_cell_sort_noalloc`) on generated
scenes of the benchmark's kind: dam-break blocks at spacing h/2 in boxes of
random aspect (`ssf_pbf_cuda_gb300/scenes.py`), the reference's own dam
parameters (h = 1.4 spacings), and its 720p frame.

Kinds:
  plain  set_particles, one_step, get_particles of one scene
  batch  step_packed and get_all_async of many scenes of uneven size
  sort   the allocation-free cell sort
  frame  one rendered frame of a particle set

Physics:
  served     the served stream's: the benchmark's configuration with s_corr
             k = 1e-4 (XSPH and vorticity confinement over the neighbour list)
  reference  the reference's active step: its own s_corr, no post passes
"""
import ctypes
import math

import numpy as np
import torch

from ssf_pbf_cuda_gb300 import _lib, api, scenes

H = 0.1         # smoothing length of the benchmark scenes
SPACING = 0.05  # h / 2


def listed():
    return [
        # the smallest request a server admits alone: one 4k scene, latency bound
        dict(name="plain_4k", kind="plain", n=4096, physics="served", boundary="planes", state="rest", iters=4),
        # the reference's dam simulator: 22^3 particles, built-in sphere, 3 iterations
        dict(name="ref_dam_10k", kind="plain", n=10648, physics="reference", boundary="sphere", state="rest", iters=3),
        # the benchmark's dam break, moving
        dict(name="plain_32k", kind="plain", n=32768, physics="served", boundary="planes", state="flow", iters=4),
        # an odd size between the small and the large steps
        dict(name="plain_150k", kind="plain", n=150001, physics="served", boundary="planes", state="flow", iters=4),
        # the single large scene
        dict(name="plain_1m", kind="plain", n=1048576, physics="served", boundary="planes", state="rest", iters=4),
        # the same size with the reference's own step (the size it is compared with the reference at)
        dict(name="ref_1m", kind="plain", n=1048576, physics="reference", boundary="planes", state="rest", iters=4),
        # what a lightly loaded server has resident
        dict(name="batch_12", kind="batch", scenes=12, n_min=8192, n_max=65536, physics="served", state="flow",
             iters=4),
        # the batched workload: 256 scenes of 4k to 64k particles
        dict(name="batch_256", kind="batch", scenes=256, n_min=4096, n_max=65536, physics="served", state="rest",
             iters=4),
        # a served mix with scenes beyond 65,536 particles
        dict(name="batch_mix", kind="batch", scenes=24, n_min=8192, n_max=262144, physics="served", state="flow",
             iters=4),
        # the allocation-free sort near its largest size, particles in random order
        dict(name="sort_250k", kind="sort", n=250007, per_cell=8.0),
        # the reference's frame: a 32k dam at 1280 x 720
        dict(name="frame_720p", kind="frame", n=32768, width=1280, height=720, mode="quad"),
        # a large set at 1920 x 1080, as point sprites
        dict(name="frame_1080p", kind="frame", n=524288, width=1920, height=1080, mode="sprite"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "batch", "batch", "batch", "sort", "frame"])
    if kind == "plain":
        physics = rng.choice(["served", "served", "reference"])
        return dict(kind=kind, n=_log_int(rng, 4096, 1048576), physics=physics, boundary="planes",
                    state=rng.choice(["rest", "flow"]), iters=rng.choice([3, 4]))
    if kind == "batch":
        n_max = rng.choice([65536, 65536, 262144])
        # at most the listed batch's particles: the mean of a log-uniform size
        # is about n_max / 3
        most = min(200, int(4.0e6 / (n_max / 3)))
        return dict(kind=kind, scenes=_log_int(rng, 2, most), n_min=rng.choice([4096, 8192]), n_max=n_max,
                    physics=rng.choice(["served", "served", "reference"]), state=rng.choice(["rest", "flow"]), iters=4)
    if kind == "sort":
        return dict(kind=kind, n=_log_int(rng, 10000, 262144), per_cell=rng.uniform(2.0, 16.0))
    w, h = rng.choice([(640, 360), (1280, 720), (1001, 563), (1920, 1080)])
    return dict(kind=kind, n=_log_int(rng, 8192, 524288), width=w, height=h, mode=rng.choice(["quad", "sprite"]))


# ----------------------------------------------------------------- inputs --

def _rng(seed, k=0):
    return np.random.Generator(np.random.PCG64(scenes.splitmix64(seed * 1000003 + k)))


def _block(n, rng, state, h=H):
    """n particles of a near-cubic lattice inside a box of random aspect with
    four times the block's volume, as the benchmark's scenes: positions,
    velocities and the box.  rest: jitter h/100 and no velocity.  flow: jitter
    3h/100 and a smooth velocity field of about 1 m/s."""
    aspect = rng.uniform(1.0, 3.0, size=3)
    box = aspect * (4.0 * n * SPACING ** 3 / float(np.prod(aspect))) ** (1.0 / 3.0)
    room = lambda b: np.maximum(1, np.floor((b - 2 * h) / SPACING).astype(int) + 1)  # noqa: E731
    dims = np.minimum(np.full(3, math.ceil(n ** (1.0 / 3.0))), room(box))
    while int(np.prod(dims)) < n:
        free = room(box) - dims
        if free.max() <= 0:
            box = box * 1.1
            continue
        dims[int(np.argmax(free))] += 1
    extent = (dims - 1) * SPACING
    lo = np.full(3, h)
    x = scenes.lattice(int(dims[0]), int(dims[1]), int(dims[2]), SPACING,
                       rng.uniform(lo, np.maximum(lo, box - h - extent)))[:n]
    jit = 0.01 * h if state == "rest" else 0.03 * h
    x = (x + rng.uniform(-jit, jit, size=x.shape)).astype(np.float32)
    if state == "rest":
        v = np.zeros_like(x)
    else:
        k, ph = rng.uniform(1.0, 3.0, size=(3, 3)), rng.uniform(0, 2 * math.pi, size=3)
        v = (0.6 * np.sin(x.astype(np.float64) @ k + ph)).astype(np.float32)
    return x, v, tuple(float(t) for t in box)


def _params(physics, box, h):
    if physics == "served":
        p = api.config_params(scorr_k=1e-4)
    else:  # the reference's dam: h = 1.4 spacings, relaxation 1 / spacing^2
        p = api.default_params(stable_distance=SPACING, particle_mass=1000.0 * SPACING ** 3, smoothing_length=h,
                               cell_width=h, relaxation=1.0 / SPACING ** 2, time_step=0.015)
    p["grid_size"] = list(api.resolve_grid(p, box))
    return p


def _scene(case, seed, k=0):
    """(x, v, params, domain end, area, planes or None) of one scene, on the host."""
    rng = _rng(seed, k)
    if case.get("boundary") == "sphere":
        # pbf_dam_sim's block in the domain [1, 10]^3, jittered so that seeds differ
        space = 0.16
        m = round(case["n"] ** (1.0 / 3.0))
        x = scenes.lattice(m, m, m, space, (2.25,) * 3)
        x = (x + rng.uniform(-0.01 * space, 0.01 * space, size=x.shape)).astype(np.float32)
        p = api.default_params(stable_distance=space, particle_mass=1000.0 * space ** 3, smoothing_length=1.4 * space,
                               cell_width=1.4 * space, relaxation=1.0 / space ** 2, time_step=0.015)
        p["grid_size"] = list(api.resolve_grid(p, (10.0,) * 3))
        return x, np.zeros_like(x), p, (10.0,) * 3, ((1.0,) * 3, (10.0,) * 3), None
    h = H if case["physics"] == "served" else 1.4 * SPACING
    n = case["n"] if case["kind"] == "plain" else _scene_size(case, k)
    x, v, box = _block(n, rng, case["state"])
    area = (tuple(-H for _ in range(3)), tuple(b + H for b in box))
    return x, v, _params(case["physics"], box, h), box, area, scenes.box_planes(box)


def _scene_size(case, k):
    """Particles of scene k of a batch: log-uniform, the same for every seed."""
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return int(round(math.exp(_rng(case["scenes"], k).uniform(lo, hi))))


def _boundary(planes):
    return None if planes is None else api.Boundary(points_on_planes=planes[0], normals_on_planes=planes[1])


def _sort_input(case, seed):
    rng = _rng(seed)
    n = case["n"]
    # cells of about per_cell particles over a power-of-two table that covers the cube
    side = (n / case["per_cell"]) ** (1.0 / 3.0)
    g = 1
    while g < side:
        g *= 2
    g = min(g, 64)
    x = rng.uniform(0.0, min(side, g) * H, size=(n, 3)).astype(np.float32)
    return x, (g, g, g)


def _frame_input(case, seed):
    """A block of particles in front of the first-frame camera, at rest spacing."""
    rng = _rng(seed)
    n = case["n"]
    m = math.ceil(n ** (1.0 / 3.0))
    s = 3.2 / m
    x = scenes.lattice(m, m, m, s, (0.4, 0.3, 0.4))[:n]
    return (x + rng.uniform(-0.05 * s, 0.05 * s, size=x.shape)).astype(np.float32)


class _DeviceImage:
    """A device image of the renderer, for torch.as_tensor.  The tensor holds
    this object and this object the renderer, whose memory the image is."""

    def __init__(self, ren, which, shape, typestr):
        self.owner = ren
        ptr = ren.image_device(which)[0]
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plain":
        x, v, p, end, area, planes = _scene(case, seed)
        part = api.PbfParticle(p, len(x), end)
        xd, vd = torch.from_numpy(x).cuda(), torch.from_numpy(v).cuda()
        return dict(kind=kind, part=part, boundary=_boundary(planes), area=area, iters=case["iters"], x=xd, v=vd,
                    x_out=torch.zeros_like(xd), v_out=torch.zeros_like(vd))
    if kind == "batch":
        sc = [_scene(case, seed, k) for k in range(case["scenes"])]
        n = sum(len(s[0]) for s in sc)
        cells = sum(int(np.prod(s[2]["grid_size"])) + 1 for s in sc)
        batch = api.Batch(len(sc), n, cells, 30)
        xd = torch.from_numpy(np.concatenate([s[0] for s in sc])).cuda()
        vd = torch.from_numpy(np.concatenate([s[1] for s in sc])).cuda()
        at = 0
        for x, _, p, end, area, planes in sc:
            batch.add_scene(p, len(x), end, _boundary(planes), area, xd[at:at + len(x)], vd[at:at + len(x)])
            at += len(x)
        return dict(kind=kind, batch=batch, iters=case["iters"], x=xd, v=vd,
                    n=np.array([len(s[0]) for s in sc], np.uint32), x_out=torch.zeros_like(xd),
                    v_out=torch.zeros_like(vd), counts=torch.zeros(len(sc), dtype=torch.int32, device="cuda"))
    if kind == "sort":
        x, g = _sort_input(case, seed)
        c = g[0] * g[1] * g[2]
        ints = lambda m: torch.zeros(m, dtype=torch.int32, device="cuda")  # noqa: E731
        return dict(kind=kind, lib=api.load(), x=torch.from_numpy(x).cuda(), grid=(ctypes.c_uint32 * 3)(*g),
                    perm=ints(len(x)), start=ints(c), end=ints(c))
    mode = _lib.PBF_SSF_SPLAT_QUAD if case["mode"] == "quad" else _lib.PBF_SSF_SPLAT_SPRITE
    ren = api.SsfRenderer(api.ssf_default_params(width=case["width"], height=case["height"], splat_mode=mode))
    w, h = ren.width, ren.height
    images = {}
    for which, shape, ts in (("depth", (h, w), "<f4"), ("normal", (h, w, 4), "<f4"), ("color", (h, w, 4), "<f4"),
                             ("rgba8", (h, w, 4), "|u1")):
        images[which] = torch.as_tensor(_DeviceImage(ren, which, shape, ts), device="cuda")
    return dict(kind=kind, ren=ren, x=torch.from_numpy(_frame_input(case, seed)).cuda(), images=images)


def run(state):
    kind = state["kind"]
    stream = torch.cuda.current_stream()
    if kind == "plain":
        part = state["part"]
        part.set_particles(state["x"], state["v"], stream)
        api.one_step(part, state["boundary"], state["area"], state["iters"], stream)
        part.get_particles_device(state["x_out"], state["v_out"], stream)
        return {"x": state["x_out"], "v": state["v_out"]}
    if kind == "batch":
        # the counts are named on each call: the scenes are loaded whole again
        state["batch"].step_packed(state["iters"], state["x"], state["v"], state["n"], stream)
        state["batch"].get_all_async(state["counts"], state["x_out"], state["v_out"], stream)
        return {"counts": state["counts"], "x": state["x_out"], "v": state["v_out"]}
    if kind == "sort":
        x = state["x"]
        _lib.check(state["lib"].pbf_cell_sort_noalloc(x.data_ptr(), x.shape[0], H, state["grid"],
                                                      state["perm"].data_ptr(), state["start"].data_ptr(),
                                                      state["end"].data_ptr(), stream.cuda_stream),
                   "pbf_cell_sort_noalloc")
        return {"perm": state["perm"], "start": state["start"], "end": state["end"]}
    state["ren"].render(state["x"], stream)
    return dict(state["images"])


def work(case):
    """Each pass of a step reads and writes its particles and cells once:
    544 B per particle and 84 B per cell at four iterations (predict and hash
    52, reorder 76, each lambda pass 36, each delta-p pass 52, velocity
    update), 160 and 24 more with XSPH and vorticity.  About 30 FP32 operations
    for each of 29 (or 11 at h = 1.4 spacings) neighbours in a pair pass."""
    kind = case["kind"]
    if kind in ("plain", "batch"):
        if kind == "plain":
            n = case["n"]
        else:
            n = sum(_scene_size(case, k) for k in range(case["scenes"]))
        served = case["physics"] == "served"
        it = case["iters"]
        cells = n / 12.0  # tables of 2h cells, rounded to powers of two
        per_n = 52 + 76 + it * 88 + 64 + 48 + (160 if served else 0)
        per_c = 20 + 16 * it + (24 if served else 0)
        pairs = 29 if served else 11
        return {"bytes": n * per_n + cells * per_c, "flops": n * pairs * 30.0 * (2 * it + (3 if served else 0))}
    if kind == "sort":
        x, g = case["n"], (case["n"] / case["per_cell"])
        return {"bytes": 12 * x + 4 * x + 8 * g, "flops": 20.0 * x}
    px = case["width"] * case["height"]
    return {"bytes": 12 * case["n"] + px * (4 + 16 + 16 + 4), "flops": 60.0 * px * 3}


# ------------------------------------------------------------------ exact --
# One step in 64 bits.  Which particle lies in which cell and which pairs are
# neighbours is decided on single-precision positions, as the interface
# defines it; everything computed from there on is in 64 bits.

def _f32(t):
    return t.to(torch.float32).to(torch.float64)


def _steps64(sc, iters, dev):
    """sc: [(x, v, params, area, planes)].  All scenes at once, particles and cells offset per scene."""
    T = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    sid = torch.cat([torch.full((len(s[0]),), k, dtype=torch.int64, device=dev) for k, s in enumerate(sc)])
    x0, v0 = T(np.concatenate([s[0] for s in sc])), T(np.concatenate([s[1] for s in sc]))
    p = dict(sc[0][2])  # physics is the same for every scene; the grid is not
    f = lambda k: float(np.float32(p[k]))  # noqa: E731
    h, m, rho, eps, dt, cw = (f(k) for k in ("smoothing_length", "particle_mass", "stable_density", "relaxation",
                                             "time_step", "cell_width"))
    h2 = float(np.float32(np.float32(h) * np.float32(h)))
    grid = torch.tensor([list(s[2]["grid_size"]) for s in sc], dtype=torch.int64, device=dev)
    ncell = grid.prod(1)
    coff = torch.cumsum(ncell, 0) - ncell
    # prediction, rounded to single precision after each fused multiply-add
    g = T(np.asarray(p["body_force"], np.float32))
    xp = _f32(_f32(g * dt + v0) * dt + x0)
    cell = torch.floor(_f32(xp / cw)).to(torch.int64)
    gp = grid[sid]
    wrap = lambda c: ((c[:, 2] % gp[:, 2]) * gp[:, 1] + c[:, 1] % gp[:, 1]) * gp[:, 0] + c[:, 0] % gp[:, 0]  # noqa: E731
    key = coff[sid] + wrap(cell)
    order = torch.sort(key, stable=True).indices
    xs, x0, v0, sid, cell, gp, key = xp[order], x0[order], v0[order], sid[order], cell[order], gp[order], key[order]
    n = len(xs)
    total = int(ncell.sum())
    start = torch.searchsorted(key, torch.arange(total + 1, device=dev))
    cap = int(p["max_pair_particle_num"]) - 1
    nb = torch.full((cap + 1, n), -1, dtype=torch.int64, device=dev)
    cnt = torch.zeros(n, dtype=torch.int64, device=dev)
    me = torch.arange(n, device=dev)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                c = cell + torch.tensor([dx, dy, dz], device=dev)
                b = coff[sid] + wrap(c)
                st, en = start[b], start[b + 1]
                for k in range(int((en - st).max()) if n else 0):
                    who = torch.nonzero((st + k < en) & (cnt < cap)).squeeze(1)
                    if not len(who):
                        break
                    j = st[who] + k
                    d = _f32(xs[who] - xs[j])
                    r2 = _f32(d[:, 2] * d[:, 2] + _f32(d[:, 1] * d[:, 1] + _f32(d[:, 0] * d[:, 0])))
                    ok = r2 < h2
                    w2, j = who[ok], j[ok]
                    nb[cnt[w2], w2] = j
                    cnt[w2] += 1
    ka, kb = 1.56668147065 / h ** 3, -14.3239448745 / h ** 4

    def pair(x, k):
        j = nb[k]
        on = j >= 0
        j = torch.where(on, j, me)
        d = x - x[j]
        r2 = (d * d).sum(1)
        r = torch.sqrt(r2)
        W = torch.where(on, ka * torch.clamp(1 - r2 / h ** 2, min=0) ** 3, torch.zeros_like(r))
        s = torch.where(on & (r > 0), kb * torch.clamp(1 - r / h, min=0) ** 2 / torch.where(r > 0, r, torch.ones_like(r)),
                        torch.zeros_like(r))
        return j, d, r, W, s

    wd = lambda q: ka * (1 - q * q) ** 3 if q <= 1 else 0.0  # noqa: E731
    x = xs.clone()
    for _ in range(iters):
        rho_sum, grad, g2 = torch.zeros(n, dtype=torch.float64, device=dev), torch.zeros_like(x), 0.0
        for k in range(cap):
            j, d, r, W, s = pair(x, k)
            rho_sum = rho_sum + W
            grad = grad + s[:, None] * d
            g2 = g2 + (s * r) ** 2
        lam = (m / rho * rho_sum - 1) / ((m / rho) ** 2 * ((grad * grad).sum(1) + g2) + eps)
        dp = torch.zeros_like(x)
        for k in range(cap):
            j, d, r, W, s = pair(x, k)
            lj = lam[j]
            if p["tensile_mode"] == _lib.PBF_TENSILE_TEXTBOOK:
                corr = f("scorr_k") * (W / wd(f("scorr_dq"))) ** int(p["scorr_n"])
            else:
                corr = 10.0 * (W / wd(0.4)) ** 4 * (torch.clamp(-lam, min=0) + torch.clamp(-lj, min=0))
            dp = dp - ((lam + lj + corr) * s)[:, None] * d
        dp = _collide64(x, m / rho * dp, sid, sc, dev)
        x = x + dp
    v = (x - x0) / dt
    mr = m / rho
    if p["vorticity_mode"] == _lib.PBF_VORTICITY_TEXTBOOK:
        w = torch.zeros_like(x)
        for k in range(cap):
            j, d, r, W, s = pair(x, k)
            w = w + torch.linalg.cross(v[j] - v, -d) * s[:, None]
        w = mr * w
        wl = torch.sqrt((w * w).sum(1))
        nv = torch.zeros_like(x)
        for k in range(cap):
            j, d, r, W, s = pair(x, k)
            nv = nv + (wl[j] * s)[:, None] * d
        nl = torch.sqrt((nv * nv).sum(1))[:, None]
        nv = torch.where(nl > 0, nv / torch.where(nl > 0, nl, torch.ones_like(nl)), torch.zeros_like(nv))
        v = v + dt * f("vc_parameter") * torch.linalg.cross(nv, w)
    if p["xsph_mode"] == _lib.PBF_XSPH_LIST:
        dv = torch.zeros_like(x)
        for k in range(cap):
            j, d, r, W, s = pair(x, k)
            dv = dv + (v[j] - v) * W[:, None]
        v = v + f("xsph_parameter") * mr * dv
    return x, v


def _collide64(x, dp, sid, sc, dev, passes=64):
    live = torch.arange(len(x), device=dev)
    sphere = sc[0][4] is None
    if not sphere:
        P = torch.as_tensor(np.stack([s[4][0] for s in sc]), dtype=torch.float64, device=dev)
        N = torch.as_tensor(np.stack([s[4][1] for s in sc]), dtype=torch.float64, device=dev)
    for _ in range(passes):
        if not len(live):
            break
        o, d, hit = x[live], dp[live].clone(), torch.zeros(len(live), dtype=torch.bool, device=dev)
        if sphere:
            c = 3.0 - (o + d)
            d2 = (c * c).sum(1)
            now = d2 > 9.0
            push = c * 1.0001 - 3.0 * c / torch.sqrt(d2)[:, None]
            d = torch.where(now[:, None], d + push, d)
            hit |= now
        else:
            for k in range(P.shape[1]):
                on, nn = P[sid[live], k], N[sid[live], k]
                q = o + d
                b, a = ((q - on) * nn).sum(1), ((o - on) * nn).sum(1)
                now = b < 0
                cross = o + (q - o) * (a.abs() / (a.abs() + b.abs()))[:, None]
                proj = q - (b / (nn * nn).sum(1))[:, None] * nn
                at = torch.where((a >= 0)[:, None], cross, proj)
                d = torch.where(now[:, None], d - ((q - at) * nn).sum(1)[:, None] * nn, d)
                hit |= now
        same = (d == dp[live]).all(1)
        dp[live] = d
        live = live[hit & ~same]
    return dp


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "sort":  # whole numbers
        x, g = _sort_input(case, seed)
        c = np.floor((x / np.float32(H)).astype(np.float32)).astype(np.int64) % np.array(g)
        key = (c[:, 2] * g[1] + c[:, 1]) * g[0] + c[:, 0]
        perm = np.argsort(key, kind="stable")
        b = np.searchsorted(key[perm], np.arange(g[0] * g[1] * g[2] + 1))
        empty = b[1:] == b[:-1]
        start, end = b[:-1].astype(np.int64), b[1:].astype(np.int64)
        start[empty], end[empty] = 0xFFFFFFFF, 0xFFFFFFFF
        i32 = lambda a: torch.from_numpy(a.astype(np.uint32).view(np.int32).copy())  # noqa: E731
        return {"perm": i32(perm), "start": i32(start), "end": i32(end)}
    if kind == "frame":
        return _frame64(case, seed)
    sc = [_scene(case, seed, k) for k in range(case.get("scenes", 1))]
    x, v = _steps64([(s[0], s[1], s[2], s[4], s[5]) for s in sc], case["iters"], dev)
    if kind == "plain":
        return {"x": x, "v": v}
    return {"counts": torch.tensor([len(s[0]) for s in sc], dtype=torch.int32), "x": x, "v": v}


def _frame64(case, seed):
    """The frame's passes in 64 bits: splat, blurs, normals, shading."""
    mode = _lib.PBF_SSF_SPLAT_QUAD if case["mode"] == "quad" else _lib.PBF_SSF_SPLAT_SPRITE
    p = api.ssf_default_params(width=case["width"], height=case["height"], splat_mode=mode)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    W, Hh = int(p["width"]), int(p["height"])
    f = lambda k: float(np.float32(p[k]))  # noqa: E731
    P = np.asarray(p["projection"], np.float64).reshape(4, 4).T  # columns in memory order
    V = np.asarray(p["view"], np.float64).reshape(4, 4).T
    PI = np.linalg.inv(P)
    T = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    x = T(_frame_input(case, seed).astype(np.float64))
    e = torch.cat([x, torch.ones_like(x[:, :1])], 1) @ T(V).T
    clip = lambda a, b: torch.stack([a, b, e[:, 2], e[:, 3]], 1) @ T(P).T  # noqa: E731
    hw, hh, rad = W * 0.5, Hh * 0.5, f("point_radius")
    quad = mode == _lib.PBF_SSF_SPLAT_QUAD
    if quad:
        r = 0.5 * rad
        lo, hi = clip(e[:, 0] - r, e[:, 1] - r), clip(e[:, 0] + r, e[:, 1] + r)
        ok = (lo[:, 2].abs() <= lo[:, 3])
        x0, y0 = lo[:, 0] / lo[:, 3] * hw + hw, lo[:, 1] / lo[:, 3] * hh + hh
        x1, y1 = hi[:, 0] / hi[:, 3] * hw + hw, hi[:, 1] / hi[:, 3] * hh + hh
        ok &= (x1 > x0) & (y1 > y0)
    else:
        size = rad * (f("point_scale") / e[:, :3].norm(dim=1))
        c = clip(e[:, 0], e[:, 1])
        ok = (c[:, :3].abs() <= c[:, 3:]).all(1) & (size > 0)
        xc, yc = c[:, 0] / c[:, 3] * hw + hw, c[:, 1] / c[:, 3] * hh + hh
        x0, x1, y0, y1 = xc - size / 2, xc + size / 2, yc - size / 2, yc + size / 2
    x0, x1, y0, y1, ez = x0[ok], x1[ok], y0[ok], y1[ok], e[ok, 2]
    depth = torch.ones(Hh * W, dtype=torch.float64, device=dev)
    i0, j0 = torch.ceil(x0 - 0.5), torch.ceil(y0 - 0.5)
    for dj in range(int((y1 - y0).max()) + 2):
        for di in range(int((x1 - x0).max()) + 2):
            cx, cy = i0 + di + 0.5, j0 + dj + 0.5
            nx, ny = (cx - x0) / (x1 - x0) * 2 - 1, (cy - y0) / (y1 - y0) * 2 - 1
            mag = nx * nx + ny * ny
            on = (cx < x1) & (cy < y1) & (cx > 0) & (cx < W) & (cy > 0) & (cy < Hh) & (mag <= 1)
            pz = ez[on] + torch.sqrt(1 - mag[on]) * rad
            d = (P[2, 2] * pz + P[2, 3]) / (P[3, 2] * pz + P[3, 3])
            at = (j0[on] + dj).long() * W + (i0[on] + di).long()
            depth.scatter_reduce_(0, at, d.clamp(0, 1), "amin")
    depth = depth.reshape(Hh, W)
    zn, zf = f("near_plane"), f("far_plane")
    linear = lambda d: 2 * zn / (zf + zn - d * (zf - zn))  # noqa: E731
    s = ((torch.arange(W, device=dev, dtype=torch.float64) + 0.5) / W).expand(Hh, W)
    t = ((torch.arange(Hh, device=dev, dtype=torch.float64) + 0.5) / Hh)[:, None].expand(Hh, W)

    def eye(s, t, d, flip):
        y = t * -2 + 1 if flip else t * 2 - 1
        c = torch.stack([s * 2 - 1, y, d, torch.ones_like(d)], -1) @ T(PI).T
        return c[..., :3] / c[..., 3:]

    def tap(img, s, t):  # bilinear with 8-bit weights, clamped to the edge
        u, v = s * W - 0.5, t * Hh - 0.5
        fu, fv = torch.floor(u), torch.floor(v)
        a, b = torch.round((u - fu) * 256) / 256, torch.round((v - fv) * 256) / 256
        at = lambda i, j: img[j.long().clamp(0, Hh - 1), i.long().clamp(0, W - 1)]  # noqa: E731
        return ((1 - a) * (1 - b) * at(fu, fv) + a * (1 - b) * at(fu + 1, fv) + (1 - a) * b * at(fu, fv + 1) +
                a * b * at(fu + 1, fv + 1))

    img = depth
    for _ in range(int(p["blur_passes"])):
        on = img != 1
        sd, td, ed = s[on], t[on], img[on]
        lin = linear(ed)
        br = f("blur_radius") * f("blur_scale") / eye(sd, td, ed, True).norm(dim=-1)
        num, den = torch.zeros_like(ed), torch.zeros_like(ed)
        for axis in (0, 1):
            for k in range(-4, 4):
                d = tap(img, sd + k * br, td) if axis == 0 else tap(img, sd, td + k * br)
                sl = linear(d)
                w = torch.exp(-(k * k) * br)
                r2 = torch.where((sl - lin).abs() < 0.01, (sl - lin) * 100, torch.zeros_like(sl))
                w = torch.where(d != 1, w * torch.exp(-r2 * r2), torch.zeros_like(w))
                num, den = num + sl * w, den + w
        num = torch.where(den > 0, num / den, num)
        out = torch.ones_like(img)
        out[on] = ((zf + zn - 2 * zn / num) / (zf - zn)).clamp(0, 1)
        img = out
    clear = T(np.asarray(p["clear_color"], np.float64))
    jj, ii = torch.meshgrid(torch.arange(Hh, device=dev), torch.arange(W, device=dev), indexing="ij")

    def eye_at(i, j):
        return eye((i + 0.5) / W, (j + 0.5) / Hh, img[j.clamp(max=Hh - 1), i.clamp(max=W - 1)], False)

    ie, je = ii - ii % 2, jj - jj % 2
    nrm = torch.linalg.cross(eye_at(ie + 1, jj) - eye_at(ie, jj), eye_at(ii, je + 1) - eye_at(ii, je))
    nrm = torch.cat([nrm / nrm.norm(dim=-1, keepdim=True), torch.ones_like(nrm[..., :1])], -1)
    nrm = torch.where((img == 1)[..., None], clear, nrm)
    light = V @ np.array([1.0, 4.0, 1.0, 0.0])
    light = T(light[:3] / np.linalg.norm(light[:3]))
    view = -eye(s, t, depth, True)
    view = view / view.norm(dim=-1, keepdim=True)
    half = light + view
    half = half / half.norm(dim=-1, keepdim=True)
    n3 = nrm[..., :3]
    spec = (half * n3).sum(-1).clamp(min=0) ** 50
    fres = 0.3 + 0.7 * (1 - (n3 * view).sum(-1)) ** 5
    diff = (light * n3).sum(-1).clamp(min=0)
    a = min(max(f("thickness"), 0.0), 1.0)
    att = T(np.exp(np.array([-5.0, -1.0, -0.1]) * a))
    rgb = (att * diff[..., None] + (spec + fres)[..., None]).clamp(0, 1) * a + clear[:3] * (1 - a)
    col = torch.cat([rgb, torch.full_like(rgb[..., :1], a * a) + clear[3] * (1 - a)], -1).clamp(0, 1)
    col = torch.where((depth == 1)[..., None], clear, col)
    return {"depth": depth, "normal": nrm, "color": col, "rgba8": None}
