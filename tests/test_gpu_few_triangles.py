"""Few triangles that cover a large grid many times over: the rasterising
voxeliser spreads them over the whole GPU, and the volumes are the oracle's
wherever the lines are cut."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import oracle as O
from helpers import GpuScene, split_records
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def _scene(n, dim, copies=1):
    rng = np.random.default_rng(n)
    tris = (rng.uniform(-0.6, 0.6, size=(n, 1, 3)) + 0.8 * rng.normal(size=(n, 3, 3))).reshape(n, 9).astype(np.float32)
    nrm = rng.normal(size=(n, 3, 3))
    nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
    many = lambda a: np.concatenate([a.astype(np.float32)] * copies)  # noqa: E731
    return dataclasses.replace(scenes.tiny(seed=n, dim=dim, gbuffer=(64, 48), shadow=256), positions=many(tris),
                               normals=many(nrm.reshape(n, 9)), albedo=many(rng.uniform(0, 1, size=(n, 3))))


@pytest.mark.parametrize("n,dim", [(1, 128), (3, 256), (255, 64), (257, 128)])
def test_volumes_match_oracle(n, dim):
    sc = _scene(n, dim)
    g = GpuScene(sc)
    count, sums, total = O.voxelize(sc, g.sm.cpu().numpy(), nthreads=8)
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc))
        ctx.voxelize_accumulate(g.tris, g.lights, g.shadow, sc.eye)
        got_count, got_sums, _, _ = split_records(*ctx.read_accumulators())
        assert ctx.stats()["total_voxel_fragments"] == total
    assert np.array_equal(got_count, count)
    assert np.array_equal(got_sums, sums.astype(np.uint32))


def test_they_fill_the_gpu():
    """Six times the triangles are six times the work: a launch that leaves no
    SM idle takes a sixth of the time, one that uses 64 CTAs most of it."""
    import torch

    def best(copies):
        sc = _scene(255, 512, copies)
        g = GpuScene(sc)
        with api.Context(api.config_for(sc)) as ctx:
            ctx.set_params(api.scene_params(sc))
            ctx.enable_timers()
            times = []
            for _ in range(8):
                ctx.frame_volume(g.tris, g.lights, g.shadow, sc.eye)
                out = g.new_outputs()
                ctx.trace(g.gb, sc.eye, api.trace_out(*out))
                torch.cuda.synchronize()
                times.append(ctx.timers()["voxelize_ms"])
        return min(times[2:])

    assert best(1) < 0.4 * best(6)
