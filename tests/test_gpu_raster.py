"""The line rasteriser of the set-up passes and of the voxeliser where its
work is split: slivers along and across the lines it walks, triangles around
the size whose edge functions leave 32 bits, triangles that fill the image or
reach far outside it, near-plane clips into two parts, triangle counts around
the CTA's 256.  The shadow map, the G-buffer and the radiance chain (lit by
point lights inside and outside their range and through a shadow map that ends
inside the volume) equal the oracle's bit for bit."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import oracle as O
from helpers import GpuScene, read_chain
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def _soup(kind: str, n: int, rng) -> np.ndarray:
    c = rng.uniform(-0.9, 0.9, size=(n, 1, 3))
    if kind == "slivers":  # thin triangles along x, y, z and diagonals, up to the volume's length
        d = rng.normal(size=(n, 3)) * 0.15 + np.eye(3)[rng.integers(0, 3, n)]
        a = rng.uniform(0.1, 1.5, size=(n, 1)) * d
        return np.stack([c[:, 0] - a, c[:, 0] + a, c[:, 0] + a + rng.normal(size=(n, 3)) * 2e-3], 1)
    if kind == "sizes":  # from under a pixel to the whole image
        s = np.exp(rng.uniform(np.log(1e-3), np.log(3.0), size=(n, 1, 1)))
        return c + s * rng.normal(size=(n, 3, 3))
    if kind == "near":  # around the camera, on both sides of its near plane
        return rng.normal(size=(n, 3, 3)) * 0.6 + np.array([0.3, 0.9, 2.4])
    far = c + rng.normal(size=(n, 3, 3)) * np.exp(rng.uniform(0.0, np.log(3e4), size=(n, 1, 1)))  # far outside
    return far


def _scene(kind: str, n: int, dim: int):
    rng = np.random.default_rng((n, len(kind)))
    base = scenes.tiny(seed=n, dim=dim, gbuffer=(321, 199), shadow=257)
    tris = _soup(kind, n, rng).reshape(n, 9).astype(np.float32)
    nrm = rng.normal(size=(n, 3, 3))
    nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
    return dataclasses.replace(base, positions=tris, normals=nrm.reshape(n, 9).astype(np.float32),
                               albedo=rng.uniform(0, 1, size=(n, 3)).astype(np.float32), shadow_size=(257, 140))


@pytest.mark.parametrize("n", [1, 31, 257, 1500])
@pytest.mark.parametrize("kind", ["slivers", "sizes", "near", "far"])
def test_depth_raster_matches_oracle(kind, n):
    sc = _scene(kind, n, 16)
    g = GpuScene(sc)
    sm, gbuf = g.host_inputs()
    assert np.array_equal(sm, O.render_shadowmap(sc))
    for got, want in zip(gbuf, O.render_gbuffer(sc)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("width", [127, 128, 129, 8192, 16384])
@pytest.mark.parametrize("kind", ["slivers", "sizes", "far"])
def test_long_lines_match_oracle(kind, width):
    """Lines around the length of a piece and beyond 64 of them."""
    sc = dataclasses.replace(_scene(kind, 67, 16), gbuffer_size=(width, 5), shadow_size=(width, 7))
    g = GpuScene(sc)
    sm, gbuf = g.host_inputs()
    assert np.array_equal(sm, O.render_shadowmap(sc))
    for got, want in zip(gbuf, O.render_gbuffer(sc)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("n,dim", [(1, 16), (31, 64), (257, 32), (1500, 128), (300, 256)])
@pytest.mark.parametrize("kind", ["slivers", "sizes", "far"])
def test_voxel_raster_matches_oracle(kind, n, dim):
    sc = _scene(kind, n, dim)
    # the shadow map covers the volume's middle only; one light far away, one whose range is 0
    half = np.diag([2.0, 2.0, 1.0, 1.0]) @ sc.ls.reshape(4, 4).T
    light = dict(position=np.array([0.1, -0.2, 0.3]), direction=np.array([0.0, -1.0, 0.0]), color=np.ones(3), range=0.5,
                 intensity=1.0, shadow_caster=1, type=0)
    extra = [light, dict(light, position=np.array([50.0, 0.0, 0.0]), shadow_caster=0), dict(light, range=0.0)]
    sc = dataclasses.replace(sc, ls=scenes.colmajor(half), ls_inverse=scenes.colmajor(np.linalg.inv(half)),
                             lights=sc.lights + extra)
    g = GpuScene(sc)
    sm, gbuf = g.host_inputs()
    ref = O.frame(sc, shadowmap=sm, gbuf=gbuf, nthreads=8)
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc))
        irr, spec, col, samples = g.new_outputs()
        ctx.frame(g.tris, g.lights, g.shadow, sc.eye, g.gb, api.trace_out(irr, spec, col, samples))
        assert np.array_equal(read_chain(ctx), ref["chain"])
        stats = ctx.stats()
    for k in ("total_voxel_fragments", "unique_voxels", "max_fragments_per_voxel"):
        assert stats[k] == ref["stats"][k]
