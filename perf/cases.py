"""Performance cases: the work a renderer built on this library has it do.

Every case goes through the public Python mirror of the C ABI (`vct_gb300.api`)
on seeded synthetic scenes of the repository's own families
(`vct_gb300.scenes`).  Kinds:

  frame    - vct_frame: the whole cone-tracing frame from resident inputs
  stages   - the same pipeline through its separate entry points, with the
             direct-light composite, as the reference's frame loop runs it
  raster   - the shadow map and G-buffer passes in front of a frame
  animate  - one frame of an animation: actors, shadow map, G-buffers of the
             viewpoints, warped and temporally filtered frame, composite
  batch    - a captured batch of scenes, replayed
  tess     - the tessellation voxeliser
  learned  - the learned indirect light and its 16-cone target
  train    - optimiser steps of the learned light's network

`exact` restates the outputs in 64-bit torch from the same inputs.  What the
entry points define on 32-bit or 16-bit values stays so there: the snapped
window coordinates that decide coverage, and the binary16 volumes.
"""

import math

import numpy as np
import torch

from vct_gb300 import _lib as L
from vct_gb300 import api, learned, scenes

DEV = "cuda:0"
FILTERS = {"software": L.VCT_FILTER_SOFTWARE, "hybrid": L.VCT_FILTER_HYBRID}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a 16^3 preview grid and a thumbnail image, where launches and the host count
        dict(name="frame_16", kind="frame", scene="tiny", dim=16, boxes=6, columns=0, segments=0, width=47, height=31,
             shadow=63, filter="software", relight=False),
        # an ordinary small scene: the Cornell box of the smoke test with the library's default sampler
        dict(name="frame_64", kind="frame", scene="cornell", dim=64, boxes=0, columns=0, segments=0, width=640,
             height=360, shadow=512, filter="software", relight=False),
        # a mid-size scene at odd sizes, with radiance relit at injection
        dict(name="frame_128_odd", kind="frame", scene="family", dim=128, boxes=1500, columns=20, segments=501,
             width=1237, height=701, shadow=1111, filter="software", relight=True),
        # the headline frame: 262,144 triangles, 256^3, 1080p, the sampler that uses the texture units
        dict(name="frame_256", kind="frame", scene="family", dim=256, boxes=4096, columns=64, segments=1664,
             width=1920, height=1080, shadow=2048, filter="hybrid", relight=False),
        # the pipeline stage by stage (voxelise, inject, mips, trace, composite), as the reference's loop calls it
        dict(name="stages_256", kind="stages", scene="family", dim=256, boxes=4096, columns=32, segments=400,
             width=1920, height=1080, shadow=2048, filter="software", relight=False),
        # the passes in front of a small frame, at odd sizes
        dict(name="raster_small", kind="raster", scene="cornell", dim=64, boxes=0, columns=0, segments=0, width=641,
             height=359, shadow=500),
        # the passes in front of the headline frame
        dict(name="raster_large", kind="raster", scene="family", dim=256, boxes=4096, columns=64, segments=1664,
             width=1920, height=1080, shadow=2048),
        # one frame of an animated scene: 64 moving actors, four viewpoints, the warp map, the temporal filter
        dict(name="animate_256", kind="animate", dim=256, actors=64, boxes=4096, columns=45, width=1280, height=720,
             shadow=2048, views=4),
        # eight scenes of uneven size served by one captured batch
        dict(name="batch_8", kind="batch", scenes=8, layout=1, shadow=1024, filter="hybrid"),
        # the reference's own default voxeliser on a mid-size scene
        dict(name="tess_256", kind="tess", dim=256, boxes=2048, columns=32, segments=832, shadow=512),
        # learned indirect light with its per-pixel fallback, and the 16-cone light it stands for
        dict(name="learned_1080p", kind="learned", dim=256, boxes=4096, columns=64, segments=1664, width=1920,
             height=1080, shadow=2048, bound=0.1),
        # training the network: four optimiser steps at the trainer's batch size, weights read back
        dict(name="train_16384", kind="train", rows=65536, batch=16384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "stages", "raster", "raster", "animate", "batch", "tess", "learned", "train"])
    size = dict(width=_log(rng, 47, 1920), height=_log(rng, 31, 1080))
    geom = dict(boxes=_log(rng, 6, 4096), columns=_log(rng, 1, 64), segments=_log(rng, 16, 1664))
    dim = rng.choice([16, 32, 64, 128, 256])
    shadow = _log(rng, 63, 2048)
    if kind in ("frame", "stages"):
        return dict(kind=kind, scene="family", dim=dim, **geom, **size, shadow=shadow,
                    filter=rng.choice(["software", "hybrid"]), relight=rng.random() < 0.3)
    if kind == "raster":
        return dict(kind=kind, scene="family", dim=dim, **geom, **size, shadow=shadow)
    if kind == "animate":
        return dict(kind=kind, dim=rng.choice([64, 128, 256]), actors=_log(rng, 1, 64), boxes=geom["boxes"],
                    columns=_log(rng, 1, 45), width=_log(rng, 160, 1280), height=_log(rng, 90, 720), shadow=shadow,
                    views=rng.randint(1, 4))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(1, 8), layout=rng.randint(2, 999), shadow=_log(rng, 256, 1024),
                    filter=rng.choice(["software", "hybrid"]))
    if kind == "tess":
        return dict(kind=kind, dim=dim, boxes=_log(rng, 6, 2048), columns=_log(rng, 1, 32), segments=_log(rng, 16, 832),
                    shadow=_log(rng, 63, 512))
    if kind == "learned":
        return dict(kind=kind, dim=rng.choice([32, 64, 128, 256]), **geom, **size, shadow=shadow,
                    bound=rng.choice([0.02, 0.05, 0.1, 0.2]))
    batch = _log(rng, 129, 16384)
    return dict(kind=kind, rows=batch * rng.randint(1, 4) + rng.randint(0, 63), batch=batch)


# ------------------------------------------------------------------ inputs
def _scene(case, seed):
    g = (case.get("width", 320), case.get("height", 180))
    s = case["shadow"]
    if case.get("scene") == "tiny":
        return scenes.tiny(seed, dim=case["dim"], shadow=s, gbuffer=g, n_boxes=case["boxes"])
    if case.get("scene") == "cornell":
        return scenes.cornell(seed, dim=case["dim"], shadow=s, gbuffer=g)
    return scenes.large_family(seed, dim=case["dim"], shadow=s, gbuffer=g, n_boxes=case["boxes"],
                               n_cyl=case["columns"], cyl_segments=case["segments"])


def _batch_scene(case, seed, k):
    """Scene k of a batch: the batched family's grids, image sizes and
    triangle counts by the layout, their contents by the seed."""
    rng = np.random.default_rng((case["layout"], k))
    dim = int(rng.choice(scenes.BATCH_DIMS))
    size = scenes.BATCH_GBUFFERS[int(rng.integers(len(scenes.BATCH_GBUFFERS)))]
    tris = math.exp(rng.uniform(math.log(1000), math.log(200000)))
    return scenes.large_family(64 * seed + k, dim=dim, shadow=case["shadow"], gbuffer=size, n_boxes=int(tris / 24),
                               n_cyl=4, cyl_segments=int(tris / 16))


def _plane(sc):
    return torch.zeros(sc.gbuffer_size[0] * sc.gbuffer_size[1] * 4, device=DEV)


def _with_room(t, rows):
    out = torch.zeros(rows, t.shape[1], device=DEV)
    out[:t.shape[0]] = t
    return out


class _Inputs:
    """A scene on the device with its shadow map and G-buffer."""

    def __init__(self, sc, rendered=True):
        self.sc = sc
        self.pos, self.nrm, self.alb = (torch.from_numpy(a).to(DEV) for a in (sc.positions, sc.normals, sc.albedo))
        self.tris = api.triangles(self.pos, self.nrm, self.alb)
        self.lights = api.light_array(sc.lights)
        (W, H), (sw, sh) = sc.gbuffer_size, sc.shadow_size
        self.sm = torch.empty(sw * sh, device=DEV)
        self.keys = torch.empty(W * H, dtype=torch.int64, device=DEV)
        self.gpos, self.gnrm, self.galb = (torch.empty(W * H * 4, device=DEV) for _ in range(3))
        self.shadow = api.shadow_desc(sc, self.sm)
        self.gb = api.gbuffer(self.gpos, self.gnrm, self.galb, W, H)
        if rendered:
            self.render()

    def render(self):
        api.render_shadowmap(self.tris, self.sc, self.sm)
        api.render_gbuffer(self.tris, self.sc, self.keys, self.gpos, self.gnrm, self.galb)


def _context(sc, **params):
    ctx = api.Context(api.config_for(sc))
    ctx.set_params(api.scene_params(sc, **params))
    return ctx


class _Volume:
    """Level 0 of a context's volume as binary16 bit patterns; a tensor made
    of it keeps the context, which owns the memory, alive."""

    def __init__(self, ctx, volume):
        ptr, d = ctx.volume_ptr(volume, 0)
        self.ctx = ctx
        self.__cuda_array_interface__ = dict(shape=(d * d * d * 4,), typestr="<i2", data=(ptr, False), version=2,
                                             strides=None)


def _volume_view(ctx, volume):
    return torch.as_tensor(_Volume(ctx, volume), device=DEV)


def _traced(sc):
    irr, spec, col = _plane(sc), _plane(sc), _plane(sc)
    return irr, spec, col, api.trace_out(irradiance=irr, specular=spec, color=col)


def _training_rows(case, seed):
    """Feature rows and 16-cone targets of random covered pixels of a scene."""
    sc = scenes.large_family(seed, dim=64, shadow=256, gbuffer=(512, 288), n_boxes=1024, n_cyl=16, cyl_segments=64)
    st = learned.FrameState(64, sc.gbuffer_size, 256)
    st.load(sc)
    st.features()
    st.reference()
    cov = torch.nonzero(st.covered()).view(-1).to(torch.int32)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    pick = cov[torch.randint(cov.numel(), (case["rows"],), generator=gen, device=DEV)].contiguous()
    rows = torch.empty(case["rows"], learned.FEATURES, device=DEV)
    st.rows(pick, rows)
    targets = st.ref.view(-1, 4)[pick.long(), :3].contiguous()
    torch.cuda.synchronize()
    st.ctx.close()
    order = torch.randperm(case["rows"], generator=gen, device=DEV).to(torch.int32)
    return rows, targets, order


def _training_rates(case):
    steps = case["rows"] // case["batch"]
    return [2e-5 + 0.5 * (2e-3 - 2e-5) * (1 + math.cos(math.pi * s / max(1, steps - 1))) for s in range(steps)]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "stages"):
        s = _Inputs(_scene(case, seed))
        s.ctx = _context(s.sc, trace_filter=FILTERS[case["filter"]], radiance_lighting=int(case["relight"]))
        s.irr, s.spec, s.col, s.out = _traced(s.sc)
        s.lit = _plane(s.sc)
        s.volumes = [_volume_view(s.ctx, v) for v in (L.VCT_VOLUME_COLOR, L.VCT_VOLUME_NORMAL)]
    elif kind == "raster":
        s = _Inputs(_scene(case, seed), rendered=False)
    elif kind == "tess":
        s = _Inputs(_scene(case, seed))
        s.ctx = _context(s.sc, voxelize_tesselation=1)
        s.volumes = [_volume_view(s.ctx, v) for v in (L.VCT_VOLUME_COLOR, L.VCT_VOLUME_NORMAL, L.VCT_VOLUME_RADIANCE)]
    elif kind == "animate":
        sc, actors = scenes.dynamic_scene(seed, n_actors=case["actors"], dim=case["dim"], shadow=case["shadow"],
                                          gbuffer=(case["width"], case["height"]), static_boxes=case["boxes"],
                                          static_cyl=case["columns"])
        s = _Inputs(sc, rendered=False)
        s.local_arrays = (s.pos, s.nrm)
        s.local = api.triangles(s.pos, s.nrm, s.alb)
        room = 12 * case["boxes"] + 3328 * case["columns"] + 8000 * case["actors"]  # the largest actors' triangles
        s.pos, s.nrm = (_with_room(t, room) for t in s.local_arrays)
        s.tris = api.triangles(s.pos, s.nrm, s.alb)
        s.tris.count = sc.ntri
        s.models = actors.models(1.0 + seed % 7)
        s.actors = api.actor_array(s.models)
        s.ctx = _context(sc, temporal_filter=1, temporal_decay=0.8, warp_mode=L.VCT_WARP_TEXTURE,
                         trace_filter=L.VCT_FILTER_HYBRID)
        s.views = [scenes.viewpoint(sc, k) for k in range(case["views"])]
        s.planes = [[_plane(sc) for _ in range(3)] for _ in s.views]
        s.gbs = [api.gbuffer(*p, *sc.gbuffer_size) for p in s.planes]
        s.irr, s.spec, s.col, s.out = _traced(sc)
        s.cols = [_plane(sc) for _ in s.views[1:]]
        s.outs = [api.trace_out(color=c) for c in s.cols]
        s.lit = _plane(sc)
    elif kind == "batch":
        s = _Batch(case, seed)
    elif kind == "learned":
        s = _Inputs(_scene(case, seed))
        s.ctx = _context(s.sc)
        s.ctx.voxelize(s.tris, s.lights, s.shadow, s.sc.eye)
        s.ctx.inject(s.shadow, s.sc.eye)
        s.ctx.build_mips()
        s.mlp = api.Mlp()
        s.mlp.set_params(learned.load_params())
        s.ref, s.pred = _plane(s.sc), _plane(s.sc)
    else:
        s = _State()
        s.rows, s.targets, s.order = _training_rows(case, seed)
        s.mlp = api.Mlp()
        s.mlp.set_params(learned.load_params())
        s.rates = _training_rates(case)
        s.loss = torch.zeros(len(s.rates), device=DEV)
    s.case = case
    return s


class _State:
    pass


class _Batch:
    def __init__(self, case, seed):
        self.scs = [_batch_scene(case, seed, k) for k in range(case["scenes"])]
        self.inputs = [_Inputs(sc) for sc in self.scs]
        self.batch = api.Batch([api.config_for(sc) for sc in self.scs])
        self.results = []
        descs = []
        for k, i in enumerate(self.inputs):
            self.batch.set_params(api.scene_params(i.sc, trace_filter=FILTERS[case["filter"]]), k)
            irr, _, col, _ = _traced(i.sc)
            self.results.append((irr, col))
            descs.append(api.scene_desc(i.tris, i.lights, i.shadow, i.sc.eye, i.gb, api.trace_out(irr, color=col)))
        self.stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        self.batch.frame(descs)
        torch.cuda.synchronize()
        self.batch.capture(descs, self.stream)


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s.case["kind"]
    if kind == "frame":
        s.ctx.frame(s.tris, s.lights, s.shadow, s.sc.eye, s.gb, s.out)
        return [s.irr, s.spec, s.col] + s.volumes
    if kind == "stages":
        s.ctx.voxelize(s.tris, s.lights, s.shadow, s.sc.eye)
        s.ctx.inject(s.shadow, s.sc.eye)
        s.ctx.build_mips()
        s.ctx.trace(s.gb, s.sc.eye, s.out)
        s.ctx.shade(s.gb, s.sc.eye, s.lights, s.shadow, s.lit, s.irr, s.spec)
        return [s.irr, s.spec, s.col, s.lit] + s.volumes
    if kind == "raster":
        s.render()
        return [s.sm, s.gpos, s.gnrm, s.galb]
    if kind == "tess":
        s.ctx.voxelize(s.tris, s.lights, s.shadow, s.sc.eye)
        return s.volumes
    if kind == "animate":
        api.transform_actors(s.local, s.actors, s.pos, s.nrm)
        api.render_shadowmap(s.tris, s.sc, s.sm)
        for v, p in zip(s.views, s.planes):
            api.render_gbuffer(s.tris, v, s.keys, *p)
        s.ctx.frame(s.tris, s.lights, s.shadow, s.views[0].eye, s.gbs[0], s.out)
        s.ctx.trace_views(s.gbs[1:], [v.eye for v in s.views[1:]], s.outs)
        s.ctx.shade(s.gbs[0], s.views[0].eye, s.lights, s.shadow, s.lit, s.irr, s.spec)
        return [s.pos, s.nrm, s.sm, s.planes[-1], s.irr, s.spec, s.col, s.lit, s.cols]
    if kind == "batch":
        s.batch.replay()
        return s.results
    if kind == "learned":
        api.trace_reference16(s.ctx, s.gb, s.sc.eye, s.ref)
        api.learned_trace_pixels(s.ctx, s.mlp, s.gb, s.sc.eye, s.pred, s.case["bound"])
        return [s.ref, s.pred]
    b = s.case["batch"]
    for k, lr in enumerate(s.rates):
        s.mlp.train_step(s.rows, s.targets, s.order[k * b:(k + 1) * b], b, lr, s.loss[k:k + 1])
    return [s.loss, s.mlp.params()]


# ------------------------------------------------------------------ the work
def _frame_work(tris, dim, pixels, shadow, planes, trace=True):
    """Triangles, shadow map and G-buffer once; colour and normal volumes and
    the radiance chain once; the output planes once.  Covered pixels (about
    0.6 of them) take some 30 cone samples of 14 RGBA lerps each."""
    vox = dim ** 3
    return dict(bytes=84.0 * tris + 4.0 * shadow * shadow + 48.0 * pixels + 16.0 * planes * pixels + 16.0 * vox +
                8.0 * vox * 8 / 7, flops=(0.6 * pixels * 30 * 14 * 4 * 3) if trace else 0.0)


def _triangles(case):
    if case.get("scene") == "cornell":
        return 1290
    return 12 * case["boxes"] + 2 * case.get("columns", 0) * case.get("segments", 0)


def work(case):
    kind = case["kind"]
    P = case.get("width", 0) * case.get("height", 0)
    if kind in ("frame", "stages"):
        return _frame_work(_triangles(case), case["dim"], P, case["shadow"], 3 if kind == "frame" else 4)
    if kind == "raster":
        return dict(bytes=84.0 * _triangles(case) + 4.0 * case["shadow"] ** 2 + 48.0 * P, flops=0.0)
    if kind == "tess":
        return _frame_work(_triangles(case), case["dim"], 0, 0, 0, trace=False)
    if kind == "animate":
        moved = 5000 * case["actors"]
        tris = 12 * case["boxes"] + 3328 * case["columns"] + moved
        w = _frame_work(tris, case["dim"], P * case["views"], case["shadow"], 1)
        w["bytes"] += 2 * 72.0 * moved + (3 + 1) * 16.0 * P + 48.0 * P * case["views"] + 4.0 * case["shadow"] ** 2
        return w
    if kind == "batch":
        w = _frame_work(40000, 160, 640 * 640, case["shadow"], 2)
        return {k: case["scenes"] * v for k, v in w.items()}
    if kind == "learned":
        return dict(bytes=(48.0 + 32.0) * P + 16.0 * case["dim"] ** 3 / 7,
                    flops=0.6 * P * (16 * 8 * 14 * 4 * 3 * 1.3 + 2 * 11332))
    n = case["rows"] // case["batch"] * case["batch"]
    return dict(bytes=n * (42 + 3 + 1) * 4.0, flops=6.0 * 11332 * n)


# ------------------------------------------------------------------ the outputs in 64 bits
def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("frame", "stages"):
            s = _Inputs(_scene(case, seed))
            chain = _chain(s, case["relight"])
            irr, spec, col = _trace(s, chain, s.gb_planes(), s.sc.eye)
            out = [irr, spec, col] + ([_shade(s, irr, spec)] if kind == "stages" else [])
            return out + [None, None]
        if kind == "raster":
            s = _Inputs(_scene(case, seed), rendered=False)
            return [_depth_map(s)] + _gbuffer(s)
        if kind == "animate":  # the moved triangles; the rest carries state through eight passes
            s = prepare(case, seed)
            s.ctx.close()
            return list(_moved(s)) + [None] * 7
        if kind == "batch":
            out = []
            for k in range(case["scenes"]):
                s = _Inputs(_batch_scene(case, seed, k))
                irr, _, col = _trace(s, _chain(s, False), s.gb_planes(), s.sc.eye)
                out.append((irr, col))
            return out
        if kind == "learned":  # the network's fallback is a decision per pixel: no value
            s = _Inputs(_scene(case, seed))
            return [_trace16(s, _chain(s, False), s.gb_planes()), None]
        if kind == "train":
            return _train(case, seed)
    return None  # whole numbers only


def _d(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV)


def _gb_planes(s):
    return [p.view(-1, 4).double() for p in (s.gpos, s.gnrm, s.galb)]


_Inputs.gb_planes = _gb_planes


def _norm(v):
    return v / v.square().sum(-1, keepdim=True).sqrt()


def _apply(m, p):
    """Column-major 4x4 times (p, 1)."""
    m = m.to(p.dtype).view(4, 4)
    return m[0] * p[..., 0:1] + m[1] * p[..., 1:2] + m[2] * p[..., 2:3] + m[3]


def _window32(clip, W, H):
    """Window coordinates in 32 bits, as coverage is defined on them."""
    ndc = clip[..., :2] / clip[..., 3:4]
    return (ndc + 1.0) * 0.5 * torch.tensor([W, H], dtype=torch.float32, device=DEV)


def _covered(win, W, H, chunk=1 << 24):
    """Pixels whose centre a triangle covers (1/256 sub-pixel grid, top-left
    rule): yields triangle, x, y and the three weights."""
    v = (win.clamp(-2.0 ** 20, 2.0 ** 20) * 256.0).round().long()
    x, y = v[..., 0], v[..., 1]
    area = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (y[:, 1] - y[:, 0]) * (x[:, 2] - x[:, 0])
    flip = (area < 0)[:, None]
    turn = torch.tensor([0, 2, 1], device=DEV)
    x, y = torch.where(flip, x[:, turn], x), torch.where(flip, y[:, turn], y)
    area = area.abs()

    def span(a, n):
        lo = -torch.div(-(a.amin(1) - 128), 256, rounding_mode="floor")
        return lo.clamp_min(0), torch.div(a.amax(1) - 128, 256, rounding_mode="floor").clamp_max(n - 1)

    (x0, x1), (y0, y1) = span(x, W), span(y, H)
    wide = (x1 - x0 + 1).clamp_min(0)
    count = torch.where(area > 0, wide * (y1 - y0 + 1).clamp_min(0), 0)
    tri = torch.nonzero(count).view(-1)
    ends = count[tri].cumsum(0)
    at, done = 0, 0
    while at < tri.numel():
        to = max(at + 1, int(torch.searchsorted(ends, done + chunk)))
        some = tri[at:to]
        t = torch.repeat_interleave(some, count[some])
        k = torch.arange(t.numel(), device=DEV) - (ends[at:to] - count[some] - done).repeat_interleave(count[some])
        px, py = x0[t] + k % wide[t], y0[t] + torch.div(k, wide[t], rounding_mode="floor")
        inside, e = torch.ones_like(t, dtype=torch.bool), []
        for i in range(3):
            a, b = (i + 1) % 3, (i + 2) % 3
            dx, dy = x[t, b] - x[t, a], y[t, b] - y[t, a]
            f = dx * (py * 256 + 128 - y[t, a]) - dy * (px * 256 + 128 - x[t, a])
            inside &= torch.where((dy < 0) | ((dy == 0) & (dx < 0)), f >= 0, f > 0)
            e.append(f)
        t, px, py = t[inside], px[inside], py[inside]
        w = torch.stack([f[inside] for f in e], 1).double() / area[t].double()[:, None]
        w = torch.where(flip[t], w[:, turn], w)
        yield t, px, py, w
        done, at = int(ends[to - 1]), to


def _lerp3(w, v):
    return (w[..., None] * v).sum(1)


def _depth_map(s):
    W, H = s.sc.shadow_size
    p = s.pos.view(-1, 3, 3)
    ls = _d(s.sc.ls)
    clip = _apply(ls, p.double())
    depth = (clip[..., 2] / clip[..., 3] + 1) * 0.5
    out = torch.ones(W * H, dtype=torch.float64, device=DEV)
    for t, px, py, w in _covered(_window32(_apply(ls, p), W, H), W, H):
        z = (w * depth[t]).sum(1)
        ok = (z >= 0) & (z <= 1)
        out.scatter_reduce_(0, (py * W + px)[ok], z[ok], "amin")
    return out


def _clip_near(c):
    """The parts of clip-space triangles in front of the near plane: their
    vertices as (n, 3, 4) and the triangles they are of."""
    d = c[..., 2] + c[..., 3]
    inside = d >= 0
    parts, owner = [c[inside.all(1)]], [torch.nonzero(inside.all(1)).view(-1)]
    for t in torch.nonzero(inside.any(1) & ~inside.all(1)).view(-1).tolist():
        poly = []
        for k in range(3):
            a, b, da, db = c[t, k], c[t, (k + 1) % 3], d[t, k], d[t, (k + 1) % 3]
            if da >= 0:
                poly.append(a)
            if (da >= 0) != (db >= 0):
                poly.append(a + da / (da - db) * (b - a))
        for f in range(1, len(poly) - 1):
            parts.append(torch.stack([poly[0], poly[f], poly[f + 1]])[None])
            owner.append(torch.tensor([t], device=DEV))
    return torch.cat(parts), torch.cat(owner)


def _gbuffer(s):
    W, H = s.sc.gbuffer_size
    p, vp = s.pos.view(-1, 3, 3), _d(s.sc.view_proj)
    clip32, owner = _clip_near(_apply(vp, p))
    clip = _clip_near(_apply(vp, p.double()))[0]
    if clip.shape[0] != clip32.shape[0]:
        clip = clip32.double()
    front = (clip32[..., 3] > 0).all(1)
    clip32, clip, owner = clip32[front], clip[front], owner[front]
    depth = (clip[..., 2] / clip[..., 3] + 1) * 0.5
    best = torch.full((W * H,), 2.0, dtype=torch.float64, device=DEV)
    hits = []
    for t, px, py, w in _covered(_window32(clip32, W, H), W, H):
        z = (w * depth[t]).sum(1)
        ok = (z >= 0) & (z <= 1)
        pix, z, t = (py * W + px)[ok], z[ok], owner[t[ok]]
        best.scatter_reduce_(0, pix, z, "amin")
        hits.append((pix, z, t))
    near = torch.full((W * H,), 1 << 40, dtype=torch.int64, device=DEV)
    for pix, z, t in hits:
        won = z <= best[pix]
        near.scatter_reduce_(0, pix[won], t[won], "amin")
    pix = torch.nonzero(near < (1 << 40)).view(-1)
    t = near[pix]
    far = torch.stack([((pix % W) + 0.5) / W * 2 - 1, (torch.div(pix, W, rounding_mode="floor") + 0.5) / H * 2 - 1,
                       torch.ones_like(pix, dtype=torch.float64)], 1).double()
    f = _apply(_d(s.sc.inv_view_proj), far)
    eye = _d(s.sc.eye)
    ray = f[:, :3] / f[:, 3:4] - eye
    v = p.double()[t]
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    pv, tv = torch.linalg.cross(ray, e2), eye - v[:, 0]
    det = (e1 * pv).sum(1)
    det = torch.where(det == 0, torch.ones_like(det), det)
    a = ((tv * pv).sum(1) / det).clamp(0, 1)
    b = ((ray * torch.linalg.cross(tv, e1)).sum(1) / det)
    b = torch.minimum(b.clamp_min(0), 1 - a)
    w = torch.stack([1 - a - b, a, b], 1)
    planes = [torch.zeros(W * H, 4, dtype=torch.float64, device=DEV) for _ in range(3)]
    planes[0][pix] = torch.cat([_lerp3(w, v), torch.ones_like(a)[:, None]], 1)
    planes[1][pix, :3] = _norm(_lerp3(w, s.nrm.view(-1, 3, 3).double()[t]))
    planes[2][pix] = torch.cat([s.alb.double()[t], torch.ones_like(a)[:, None]], 1)
    return [q.view(-1) for q in planes]


def _moved(s):
    pos, nrm = (a.double().view(-1, 3, 3) for a in s.local_arrays)
    pos, nrm = pos.clone(), nrm.clone()
    room = s.pos.shape[0]
    for k, (first, count, _) in enumerate(s.models):
        m = _d(np.ctypeslib.as_array(s.actors[0][k].model))
        at = slice(first, first + count)
        pos[at] = _apply(m, pos[at])[..., :3]
        nrm[at] = nrm[at] @ torch.linalg.inv(m.view(4, 4)[:3, :3].T)
    full = [torch.zeros(room, 9, dtype=torch.float64, device=DEV) for _ in range(2)]
    for f, a in zip(full, (pos, nrm)):
        f[:a.shape[0]] = a.view(-1, 9)
    return full


def _shadow_bilinear(s, u, v, ox=0, oy=0):
    W, H = s.sc.shadow_size
    x, y = u * W + ox - 0.5, v * H + oy - 0.5
    i, j = x.floor(), y.floor()
    a, b = x - i, y - j
    sm = s.sm.double()

    def at(i, j):
        ok = (i >= 0) & (j >= 0) & (i < W) & (j < H)
        k = (j.clamp(0, H - 1) * W + i.clamp(0, W - 1)).long()
        return torch.where(ok, sm[k], torch.ones_like(a))

    low = at(i, j) * (1 - a) + at(i + 1, j) * a
    return low * (1 - b) + (at(i, j + 1) * (1 - a) + at(i + 1, j + 1) * a) * b


def _shadowed(s, p):
    c = _apply(_d(s.sc.ls), p)
    c = (c[..., :3] / c[..., 3:4] + 1) * 0.5
    z = c[..., 2] - 0.01
    f = sum((z > _shadow_bilinear(s, c[..., 0], c[..., 1], ox, oy)).double()
            for ox, oy in ((0, 0), (1, 0), (0, 1), (-1, 0), (0, -1))) / 5
    return torch.where(z > 1, torch.zeros_like(f), f)


def _attenuation(light, dist):
    t = ((dist - 0.75 * light["range"]) / (0.25 * light["range"])).clamp(0, 1)
    return 1 - t * t * (3 - 2 * t)


def _half(v):
    return v.half().double()


def _chain(s, relight):
    """The radiance chain: voxelise, average, inject, box-filter, each level
    stored binary16.  A list of (z, y, x, rgba) tensors."""
    sc, N = s.sc, s.sc.dim
    p, n = s.pos.view(-1, 3, 3), s.nrm.view(-1, 3, 3)
    face = _norm(n.sum(1)).abs()
    axis = torch.where((face[:, 0] > face[:, 1]) & (face[:, 0] > face[:, 2]), 0,
                       torch.where((face[:, 1] > face[:, 0]) & (face[:, 1] > face[:, 2]), 1, 2))
    mvp = _voxel_matrices(sc.vmax)
    sums = torch.zeros(N ** 3, 7, dtype=torch.int64, device=DEV)
    for ax in range(3):
        own = torch.nonzero(axis == ax).view(-1)
        if not own.numel():
            continue
        clip = _apply(mvp[ax], p[own])
        z = _apply(mvp[ax].double(), p[own].double())[..., 2]
        for t, px, py, w in _covered(_window32(clip, N, N), N, N):
            zf = (w * z[t]).sum(1)
            depth = (N * (1 - (zf + 1) * 0.5)).long()
            v = {0: (depth, py, N - 1 - px), 1: (px, depth, N - 1 - py), 2: (px, py, depth)}[ax]
            ok = (zf >= -1) & (zf <= 1) & (depth >= 0) & (depth < N)
            g = own[t[ok]]
            at = ((v[2] * N + v[1]) * N + v[0])[ok]
            wp, nf = _lerp3(w[ok], p.double()[g]), _norm(_lerp3(w[ok], n.double()[g]))
            val = torch.cat([_voxel_light(s, s.alb.double()[g], wp, nf), (nf + 1) * 0.5], 1)
            q = (val.clamp(0, 1) * 65535).round().long()
            sums.index_add_(0, at, torch.cat([torch.ones_like(at)[:, None], q], 1))
    count = sums[:, 0:1]
    mean = _half(sums[:, 1:] / (65535.0 * count.clamp_min(1)))
    full = (count > 0).double()
    color = torch.cat([mean[:, :3], 0.5 * full], 1)
    rad = torch.cat([torch.zeros_like(mean[:, :3]), 0.5 * full], 1)
    lit = _lit_voxels(s, N)
    if relight:
        at = torch.stack([lit % N, torch.div(lit, N, rounding_mode="floor") % N,
                          torch.div(lit, N * N, rounding_mode="floor")], 1).double()
        lv = (_d(sc.light_pos) + sc.vmax) / (2 * sc.vmax) * N
        nn = 2 * torch.where(count[lit] > 0, mean[lit, 3:], torch.zeros_like(at)) - 1
        diff = (nn * _norm(lv - at)).sum(1, keepdim=True).clamp_min(0)
        rad[lit] = _half(torch.cat([diff * _d(sc.light_int) * color[lit, :3], color[lit, 3:]], 1))
    else:
        rad[lit] = color[lit]
    levels = [rad.view(N, N, N, 4)]
    while len(levels) < sc.levels:
        a = levels[-1]
        h = a.shape[0] // 2
        levels.append(_half(a.view(h, 2, h, 2, h, 2, 4).mean((1, 3, 5))))
    return levels


def _voxel_matrices(vmax):
    """The three orthographic views of the volume, in 32 bits."""
    e = vmax
    out = []
    for eye, up in (((e, 0, 0), (0, 1, 0)), ((0, e, 0), (0, 0, -1)), ((0, 0, e), (0, 1, 0))):
        m = scenes.ortho(-e, e, -e, e, 0.0, 2 * e) @ scenes.look_at(eye, (0, 0, 0), up)
        out.append(torch.from_numpy(scenes.colmajor(m)).to(DEV))
    return out


def _voxel_light(s, color, p, n):
    total = torch.zeros_like(color)
    for light in s.sc.lights:
        col = color * _d(light["color"]).float().double() * float(np.float32(light["intensity"]))
        if light["type"] == 0:
            d = _d(light["position"]).float().double() - p
            dist = d.square().sum(1, keepdim=True).sqrt()
            lit = col * (n * d / dist).sum(1, keepdim=True).clamp_min(0) * _attenuation(light, dist)
        else:
            lit = col * (n * _norm(-_d(light["direction"]))).sum(1, keepdim=True).clamp_min(0)
        if light["shadow_caster"]:
            lit = lit * (1 - _shadowed(s, p))[:, None]
        total = total + lit
    return total.clamp(0, 1)


def _lit_voxels(s, N):
    W, H = s.sc.shadow_size
    nx, ny = min((W + 15) // 16 * 16, W + 1), min((H + 15) // 16 * 16, H + 1)
    u = (torch.arange(nx, device=DEV).double() / W).repeat(ny)
    v = (torch.arange(ny, device=DEV).double() / H).repeat_interleave(nx)
    ndc = torch.stack([u, v, _shadow_bilinear(s, u, v)], 1) * 2 - 1
    w = _apply(_d(s.sc.ls_inverse), ndc)[:, :3]
    t = ((w + s.sc.vmax) / (2 * s.sc.vmax) * N)
    i = t.long()
    i = i[((i >= 0) & (i < N)).all(1)]
    return torch.unique((i[:, 2] * N + i[:, 1]) * N + i[:, 0])


def _sample(chain, p, lod):
    """GL_LINEAR_MIPMAP_LINEAR with a zero border; lod is one number > 0."""
    top = len(chain) - 1

    def level(l):
        a = chain[l]
        S = a.shape[0]
        u = p * S - 0.5
        f = u.floor()
        w, f = u - f, f.long()
        out = torch.zeros(p.shape[0], 4, dtype=torch.float64, device=DEV)
        flat = a.view(-1, 4)
        for k in range(8):
            o = torch.tensor([k & 1, (k >> 1) & 1, k >> 2], device=DEV)
            c = f + o
            ok = ((c >= 0) & (c < S)).all(1)
            c = c.clamp(0, S - 1)
            wt = torch.where(o.bool(), w, 1 - w).prod(1) * ok
            out += wt[:, None] * flat[(c[:, 2] * S + c[:, 1]) * S + c[:, 0]]
        return out

    if lod >= top:
        return level(top)
    fine = int(math.floor(lod))
    f = lod - fine
    return level(fine) * (1 - f) + level(fine + 1) * f


def _cone(chain, start_pos, n, d, setting, N):
    """traceCone: front to back, to opacity 0.95, the volume's edge, its diagonal or the step limit."""
    steps, angle, bias, h, offset = setting
    tan = math.tan(float(np.float32(angle)) * 0.5)
    d = _norm(d)
    start = start_pos + n * bias / N
    acc = torch.zeros(n.shape[0], 4, dtype=torch.float64, device=DEV)
    live = torch.arange(n.shape[0], device=DEV)
    for _ in range(steps):
        if h / N > math.sqrt(3.0) or not live.numel():
            break
        r = h * tan
        p = start[live] + d[live] * (h / N)
        ok = ((p >= 0) & (p <= 1)).all(1)
        live, p = live[ok], p[ok]
        v = _sample(chain, p, math.log2(max(1.0, 2 * r)) + offset)
        acc[live] += (1 - acc[live, 3:]) * v
        live = live[acc[live, 3] < 0.95]
        h += r
    return acc


_DIFFUSE = ((0, 1, 0, .25), (0, .5, .866025, .15), (.823639, .5, .267617, .15), (.509037, .5, -.700629, .15),
            (-.5909037, .5, -.700629, .15), (-.823639, .5, .267617, .15))


def _frame_of(n):
    sg = torch.where(n[:, 2] >= 0, 1.0, -1.0).double()
    a = -1 / (sg + n[:, 2])
    b = n[:, 0] * n[:, 1] * a
    return (torch.stack([1 + sg * n[:, 0] ** 2 * a, sg * b, -sg * n[:, 0]], 1),
            torch.stack([b, sg + n[:, 1] ** 2 * a, -n[:, 1]], 1))


def _per_pixel(s, planes, fn, count, chunk=1 << 18):
    """fn over the covered pixels, a chunk at a time, into `count` float4 planes."""
    pix = torch.nonzero(planes[0][:, 3] != 0).view(-1)
    out = [torch.zeros(planes[0].shape[0], 4, dtype=torch.float64, device=DEV) for _ in range(count)]
    for at in range(0, pix.numel(), chunk):
        k = pix[at:at + chunk]
        for o, v in zip(out, fn(k, [q[k] for q in planes])):
            o[k] = v
    return [o.view(-1) for o in out]


def _tone(rgb):
    return torch.cat([(rgb / (rgb + 1)) ** (1 / 2.2), torch.ones_like(rgb[:, :1])], 1)


def _trace(s, chain, planes, eye):
    sc, N = s.sc, s.sc.dim
    eye = _d(eye)

    def pixels(_, g):
        n = _norm(g[1][:, :3])
        vp = (g[0][:, :3] + sc.vmax) / (2 * sc.vmax)
        t, b = _frame_of(n)
        irr = 0
        for x, y, z, w in _DIFFUSE:
            x, y, z, w = (float(np.float32(c)) for c in (x, y, z, w))
            irr = irr + w * _cone(chain, vp, n, t * x + n * y - b * z, sc.cone["diffuse"], N)
        i = g[0][:, :3] - eye
        spec = _cone(chain, vp, n, i - n * 2 * (n * i).sum(1, keepdim=True), sc.cone["specular"], N)
        rgb = (irr[:, :3] + spec[:, :3]) * g[2][:, :3] * (1 - irr[:, 3:].clamp(0, 1))
        return irr, spec, _tone(rgb)

    return _per_pixel(s, planes, pixels, 3)


def _trace16(s, chain, planes):
    i = np.arange(16)
    z = 1 - (i + 0.5) / 16
    r, phi = np.sqrt(1 - z * z), np.pi * (3 - np.sqrt(5)) * i
    dirs = np.stack([r * np.cos(phi), r * np.sin(phi), z, z / z.sum()], 1).astype(np.float32).astype(np.float64)
    _, _, bias, h, offset = s.sc.cone["diffuse"]
    cone = (24, float(np.float32(2 * np.arccos(15 / 16))), bias, h, offset)

    def pixels(_, g):
        n = _norm(g[1][:, :3])
        vp = (g[0][:, :3] + s.sc.vmax) / (2 * s.sc.vmax)
        t, b = _frame_of(n)
        acc = sum(w * _cone(chain, vp, n, t * x + b * y + n * zz, cone, s.sc.dim) for x, y, zz, w in dirs)
        return (torch.cat([acc[:, :3], torch.zeros_like(acc[:, :1])], 1),)

    return _per_pixel(s, planes, pixels, 1)[0]


def _shade(s, irr, spec):
    """phong.frag's composite: Cook-Torrance at roughness 0.5, metallic 0."""
    pi = float(np.float32(3.1415982))
    irr, spec = irr.view(-1, 4), spec.view(-1, 4)
    dot = lambda a, b: (a * b).sum(1, keepdim=True)  # noqa: E731

    def pixels(k, g):
        p, n, dc = g[0][:, :3], _norm(g[1][:, :3]), g[2][:, :3]
        v = _norm(_d(s.sc.eye) - p)
        total = torch.zeros_like(p)
        for light in s.sc.lights:
            lc = _d(light["color"]).float().double()
            if light["type"] == 0:
                d = _d(light["position"]).float().double() - p
                dist = d.square().sum(1, keepdim=True).sqrt()
                l, att = d / dist, _attenuation(light, dist) * (dist <= light["range"])
            else:
                l, att = _norm(-_d(light["direction"]))[None].expand_as(p), 1.0
            h = _norm(v + l)
            nl, nv, nh, hv = (dot(a, b).clamp_min(0) for a, b in ((n, l), (n, v), (n, h), (h, v)))
            d_ = 0.25 / (pi * (nh ** 2 * (0.25 - 1) + 1) ** 2)
            kk = 1.5 ** 2 / 8
            geo = nv / (nv * (1 - kk) + kk) * nl / (nl * (1 - kk) + kk)
            f = 0.04 + 0.96 * (1 - hv) ** 5
            out = lc * nl * ((1 - f) * dc / pi + d_ * geo * f / (4 * nl * nv).clamp_min(0.001)) * att
            if light["shadow_caster"]:
                out = out * (1 - _shadowed(s, p))[:, None]
            total = total + out
        rgb = ((irr[k, :3] + spec[k, :3]) * dc + total) * (1 - irr[k, 3:].clamp(0, 1))
        return (_tone(rgb),)

    return _per_pixel(s, s.gb_planes(), pixels, 1)[0]


def _train(case, seed):
    """The optimiser steps with a 64-bit network and 64-bit Adam."""
    rows, targets, order = _training_rows(case, seed)
    sizes = [(64, 42), (64,), (64, 64), (64,), (64, 64), (64,), (4, 64), (4,)]
    flat = _d(learned.load_params())
    at, w = 0, []
    for shape in sizes:
        n = math.prod(shape)
        w.append(flat[at:at + n].view(shape).clone().requires_grad_())
        at += n
    m, v, losses, b = [torch.zeros_like(x) for x in w], [torch.zeros_like(x) for x in w], [], case["batch"]
    for step, lr in enumerate(_training_rates(case), 1):
        pick = order[(step - 1) * b:step * b].long()
        with torch.enable_grad():
            h = rows[pick].double()
            for k in range(3):
                h = torch.relu(h @ w[2 * k].T + w[2 * k + 1])
            y = h @ w[6].T + w[7]
            e = y[:, :3] - targets[pick].double()
            loss = e.square().mean() + 0.5 * (y[:, 3] - e.square().sum(1).sqrt().detach()).square().mean()
        losses.append(loss.detach())
        for k, g in enumerate(torch.autograd.grad(loss, w)):
            m[k] = 0.9 * m[k] + 0.1 * g
            v[k] = 0.999 * v[k] + 0.001 * g * g
            w[k].data -= lr * (m[k] / (1 - 0.9 ** step)) / ((v[k] / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return [torch.stack(losses), torch.cat([x.detach().view(-1) for x in w])]
