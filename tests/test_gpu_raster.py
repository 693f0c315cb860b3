"""The depth rasteriser of the set-up passes where its work is split: slivers
along and across the lines it walks, triangles around the size that is left to
the whole CTA, triangles that fill the image or reach far outside it,
near-plane clips into two parts, triangle counts around the CTA's 256.  The
shadow map and the G-buffer equal the oracle's bit for bit."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import oracle as O
from helpers import GpuScene
from vct_gb300 import scenes

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


@pytest.mark.parametrize("n", [1, 31, 257, 1500])
@pytest.mark.parametrize("kind", ["slivers", "sizes", "near", "far"])
def test_depth_raster_matches_oracle(kind, n):
    rng = np.random.default_rng((n, len(kind)))
    base = scenes.tiny(seed=n, gbuffer=(321, 199), shadow=257)
    tris = _soup(kind, n, rng).reshape(n, 9).astype(np.float32)
    nrm = rng.normal(size=(n, 3, 3))
    nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
    sc = dataclasses.replace(base, positions=tris, normals=nrm.reshape(n, 9).astype(np.float32),
                             albedo=rng.uniform(0, 1, size=(n, 3)).astype(np.float32), shadow_size=(257, 140))
    g = GpuScene(sc)
    sm, gbuf = g.host_inputs()
    assert np.array_equal(sm, O.render_shadowmap(sc))
    for got, want in zip(gbuf, O.render_gbuffer(sc)):
        assert np.array_equal(got, want)
