"""Triangles whose edges cross the image from one end of the snapped coordinates'
range to the other (2^28 sub-pixel units, where fp32 holds a crossing to
some 240 of them): the depth passes and the rasterising voxeliser equal the
oracle's exact edge functions bit for bit."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import oracle as O
from helpers import GpuScene, split_records
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def _scene(reach, n, size, dim=16):
    """n triangles through the volume, `reach` long on both sides of it: thin
    ones, half-planes, and strips whose long edges lie in the image."""
    rng = np.random.default_rng((n, int(reach)))
    c = rng.uniform(-0.8, 0.8, size=(n, 3))
    d = rng.normal(size=(n, 3))
    d[::4] = np.eye(3)[rng.integers(0, 3, len(d[::4]))] + rng.normal(size=(len(d[::4]), 3)) * 1e-4  # nearly along an axis
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    wide = np.exp(rng.uniform(np.log(1e-3), np.log(reach), size=(n, 1)))
    a, b = c - reach * rng.uniform(0.2, 1.0, (n, 1)) * d, c + reach * rng.uniform(0.2, 1.0, (n, 1)) * d
    tris = np.stack([a, b, b + wide * rng.normal(size=(n, 3))], 1)
    nrm = rng.normal(size=(n, 3, 3))
    nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
    return dataclasses.replace(scenes.tiny(seed=n, dim=dim, gbuffer=size, shadow=64), shadow_size=size,
                               positions=tris.reshape(n, 9).astype(np.float32), normals=nrm.reshape(n, 9).astype(np.float32),
                               albedo=rng.uniform(0, 1, size=(n, 3)).astype(np.float32))


@pytest.mark.parametrize("size", [(64, 257), (1021, 63), (16384, 3)])
@pytest.mark.parametrize("reach", [30.0, 1e3, 1e5])
def test_depth_passes(reach, size):
    sc = _scene(reach, 300, size)
    g = GpuScene(sc)
    sm, gbuf = g.host_inputs()
    assert np.array_equal(sm, O.render_shadowmap(sc))
    for got, want in zip(gbuf, O.render_gbuffer(sc)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("reach,dim", [(1e3, 64), (1e5, 32), (1e5, 256)])
def test_voxeliser(reach, dim):
    sc = _scene(reach, 300, (64, 64), dim)
    g = GpuScene(sc)
    count, sums, total = O.voxelize(sc, g.sm.cpu().numpy(), nthreads=8)
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc))
        ctx.voxelize_accumulate(g.tris, g.lights, g.shadow, sc.eye)
        got_count, got_sums, _, _ = split_records(*ctx.read_accumulators())
        assert ctx.stats()["total_voxel_fragments"] == total
    assert count.any() and np.array_equal(got_count, count) and np.array_equal(got_sums, sums.astype(np.uint32))
