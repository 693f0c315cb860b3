"""Lights whose colour or intensity is not a finite number, in the rasterising
voxeliser: a fragment out of a point light's range, or turned away from it,
gets NaN from NaN x 0 and infinity x 0 all the same (and the stored colour 0 in
that component).  Accumulators equal the oracle's."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import oracle as O
from helpers import GpuScene, split_records
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu

nan, inf = float("nan"), float("inf")


@pytest.mark.parametrize("black", [False, True], ids=["albedo", "black_in_green"])
@pytest.mark.parametrize("light", [dict(color=np.array([nan, 1.0, 1.0])), dict(color=np.array([1.0, nan, nan])),
                                   dict(color=np.array([1.0, inf, 0.5])), dict(intensity=nan), dict(intensity=inf)],
                         ids=["nan_red", "nan_green_blue", "inf_green", "nan_intensity", "inf_intensity"])
def test_lights_without_a_finite_colour(light, black):
    sc = scenes.cornell(seed=5, dim=32, gbuffer=(32, 18))
    point = dict(position=np.array([0.1, -0.2, 0.3]), direction=np.array([0.0, -1.0, 0.0]), color=np.ones(3), range=0.5,
                 intensity=1.0, shadow_caster=0, type=0)
    sun = dict(point, type=1, color=np.array([0.7, 0.8, 0.9]))
    albedo = sc.albedo.copy()
    if black:
        albedo[::2, 1] = 0.0
    sc = dataclasses.replace(sc, lights=[sun, dict(point, **light)], albedo=albedo)
    g = GpuScene(sc)
    count, sums, total = O.voxelize(sc, g.sm.cpu().numpy(), nthreads=4)
    assert count.any()
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc))
        ctx.voxelize_accumulate(g.tris, g.lights, g.shadow, sc.eye)
        got_count, got_sums, occ, pad = split_records(*ctx.read_accumulators())
    assert np.array_equal(got_count, count)
    assert np.array_equal(got_sums.astype(np.uint64), sums)
