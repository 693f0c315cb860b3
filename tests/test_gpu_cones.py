"""The cone march around the size of its step table (64 steps a cone), for each
of its variants (no warp, the warp map, any warp): irradiance, specular light
and sample counts against the fp32 oracle."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from helpers import GpuScene, rel_l2, rgb
from vct_gb300 import _lib as L
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warp", [L.VCT_WARP_NONE, L.VCT_WARP_TEXTURE, L.VCT_WARP_ANALYTIC])
@pytest.mark.parametrize("steps", [1, 63, 64, 65, 150])
def test_cone_steps_match_oracle(steps, warp):
    sc = scenes.cornell(seed=3, gbuffer=(61, 35))
    # narrow cones, so that every step of the longest one is inside the volume
    sc.cone = dict(diffuse=(steps, 0.04, 1.0, 1.0, 0.5), specular=(steps, 0.05, 1.7, 0.5, 0.1))
    g = GpuScene(sc)
    sm, gbuf = g.host_inputs()
    ref = O.frame(sc, shadowmap=sm, gbuf=gbuf, nthreads=4, warp_mode=warp)
    ctx = api.Context(api.config_for(sc))
    ctx.set_params(api.scene_params(sc, warp_mode=warp))
    irr, spec, col, samples = g.new_outputs()
    ctx.frame(g.tris, g.lights, g.shadow, sc.eye, g.gb, api.trace_out(irr, spec, col, samples))
    # A distance after n steps is off by 2 n 2^-24 at most (two roundings a
    # step), a level by that / ln 2, i.e. 3e-5 at 150 steps, and a sample by
    # no more of its value; as much again for the other roundings of a step.
    assert rel_l2(rgb(irr.cpu().numpy()), rgb(ref["irradiance"])) <= 1e-4
    assert rel_l2(rgb(spec.cpu().numpy()), rgb(ref["specular"])) <= 1e-4
    assert int(samples.item()) == pytest.approx(ref["samples"], rel=1e-3)
    ctx.close()
