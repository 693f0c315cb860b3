"""The tessellation voxeliser's two kernels: the walk of slivers, for scenes
that consist of them, and single points for all others.  Accumulators and
point counts of scenes on either side equal the oracle's, sums past 2^32
included, and so do batches of them; and ordinary triangles cost about as much a
point as slivers do."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import oracle as O
from helpers import GpuScene, split_records
from vct_gb300 import _lib as L
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def _soup(n, dim, size):
    rng = np.random.default_rng(n)
    tris = (rng.uniform(-0.8, 0.8, size=(n, 1, 3)) + size * rng.normal(size=(n, 3, 3))).reshape(n, 9)
    nrm = rng.normal(size=(n, 3, 3))
    nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
    return dataclasses.replace(scenes.tiny(seed=n, dim=dim, gbuffer=(64, 48), shadow=64), positions=tris.astype(np.float32),
                               normals=nrm.reshape(n, 9).astype(np.float32),
                               albedo=rng.uniform(0, 1, size=(n, 3)).astype(np.float32))


def _family(dim, boxes, columns, segments):
    return scenes.large_family(3, dim=dim, shadow=64, gbuffer=(64, 48), n_boxes=boxes, n_cyl=columns, cyl_segments=segments)


SCENES = {
    "one": lambda: _soup(1, 64, 0.8), "a_few": lambda: _soup(33, 256, 0.5), "blocks": lambda: _soup(513, 32, 0.1),
    "boxes": lambda: _family(64, 700, 1, 16),          # few of the points are slivers'
    "few_slivers": lambda: _family(64, 20, 3, 64),     # nearly all, but of few
    "columns": lambda: _family(16, 30, 4, 832),        # inner levels of 16
    "columns_64": lambda: _family(64, 20, 4, 300),     # of 64
    "half": lambda: _family(128, 1200, 6, 64),         # boxes between the slivers
}


@pytest.mark.parametrize("warp", [L.VCT_WARP_NONE, L.VCT_WARP_PERSPECTIVE], ids=["linear", "perspective"])
@pytest.mark.parametrize("name", SCENES)
def test_accumulators_match_oracle(name, warp):
    sc = SCENES[name]()
    g = GpuScene(sc)
    count, sums, total = O.voxelize_tess(sc, nthreads=8, warp=O.warp(sc, warp) if warp else None)
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc, voxelize_tesselation=1, warp_mode=warp))
        ctx.voxelize_accumulate(g.tris, g.lights, g.shadow, sc.eye)
        got_count, got_sums, occ, pad = split_records(*ctx.read_accumulators())
        assert ctx.stats()["total_voxel_fragments"] == total
    assert np.array_equal(got_count, count) and np.array_equal(occ, count > 0)
    assert np.array_equal(got_sums.astype(np.uint64), sums) and np.all(pad == 0)


def test_single_points_past_65536_in_a_voxel():
    """30,000 copies of a triangle of a voxel's size: no slivers, so single points."""
    one = _soup(1, 16, 0.01)
    s = 2.0 / 16
    tri = np.array([0.1, 0.1, 0.1, 1.3, 0.2, 0.3, 0.4, 1.2, 0.5]) * s
    sc = dataclasses.replace(one, positions=np.repeat(tri[None], 30000, 0).astype(np.float32),
                             normals=np.repeat(one.normals, 30000, 0), albedo=np.full((30000, 3), 1.0, dtype=np.float32))
    count, sums, total = O.voxelize_tess(sc, nthreads=8)
    assert count.max() > 65537 and sums.max() >= 2 ** 32
    color, normal, _, _ = O.normalize(sc, count, sums)
    g = GpuScene(sc)
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc, voxelize_tesselation=1))
        ctx.voxelize(g.tris, g.lights, g.shadow, sc.eye)
        got = [ctx.read_volume(v, 0).cpu().numpy().view(np.uint16) for v in (L.VCT_VOLUME_COLOR, L.VCT_VOLUME_NORMAL)]
        stats = ctx.stats()
    assert np.array_equal(got[0], color) and np.array_equal(got[1], normal)
    assert stats["error_flags"] == 0 and stats["total_voxel_fragments"] == total


@pytest.mark.parametrize("names", [("boxes", "one", "few_slivers"), ("columns", "boxes"), ("blocks", "columns_64", "one")])
def test_batches_match_oracle(names):
    scs = [SCENES[n]() for n in names]
    gs = [GpuScene(sc) for sc in scs]
    batch = api.Batch([api.config_for(sc) for sc in scs])
    for i, sc in enumerate(scs):
        batch.set_params(api.scene_params(sc, voxelize_tesselation=1), i)
    outs = [g.new_outputs() for g in gs]
    batch.frame([api.scene_desc(g.tris, g.lights, g.shadow, sc.eye, g.gb, api.trace_out(*o))
                 for sc, g, o in zip(scs, gs, outs)])
    for sc, ctx in zip(scs, batch.scenes):
        count, sums, total = O.voxelize_tess(sc, nthreads=8)
        color, normal, _, st = O.normalize(sc, count, sums)
        assert np.array_equal(ctx.read_volume(L.VCT_VOLUME_COLOR, 0).cpu().numpy().view(np.uint16), color)
        assert np.array_equal(ctx.read_volume(L.VCT_VOLUME_NORMAL, 0).cpu().numpy().view(np.uint16), normal)
        stats = ctx.stats()
        assert stats["total_voxel_fragments"] == total and stats["unique_voxels"] == st["unique_voxels"]
    batch.close()


def test_ordinary_triangles_cost_no_more_than_slivers():
    """2,048 boxes in 64^3, 1.2 M points, against 286 boxes and four columns of
    64 segments, 1.6 M: the time a point is of the same size (it was three
    times as long when the boxes' were walked too)."""
    import torch

    def per_point(boxes, columns, segments):
        sc = _family(64, boxes, columns, segments)
        g = GpuScene(sc)
        with api.Context(api.config_for(sc)) as ctx:
            ctx.set_params(api.scene_params(sc, voxelize_tesselation=1))
            ctx.enable_timers()
            out, times = g.new_outputs(), []
            for _ in range(12):
                ctx.frame_volume(g.tris, g.lights, g.shadow, sc.eye)
                ctx.trace(g.gb, sc.eye, api.trace_out(*out))
                torch.cuda.synchronize()
                times.append(ctx.timers()["voxelize_ms"])
            return min(times[2:]) / ctx.stats()["total_voxel_fragments"]

    assert per_point(2048, 1, 16) < 2.0 * per_point(286, 4, 64)
