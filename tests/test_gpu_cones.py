"""The cone march around the size of its step table (64 steps a cone), for each
of its variants (no warp, the warp map, any warp): irradiance, specular light
and sample counts against the fp32 oracle; and the tracer's two kernels against each other."""

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


@pytest.mark.parametrize("filt", [L.VCT_FILTER_SOFTWARE, L.VCT_FILTER_HYBRID])
def test_few_and_many_pixels_give_the_same_bits(filt):
    """An image of 5,000 tiles (a warp to 32 pixels) and its bands of 20 to 1,120
    tiles (four warps; two steps at a time up to 38 tiles): every output, and
    the number of samples."""
    import torch

    W, H = 317, 3990
    sc = scenes.cornell(seed=4, gbuffer=(W, H))
    g = GpuScene(sc)
    ctx = api.Context(api.config_for(sc))
    ctx.set_params(api.scene_params(sc, trace_filter=filt))
    ctx.frame_volume(g.tris, g.lights, g.shadow, sc.eye)
    whole, bands = g.new_outputs(), g.new_outputs()
    ctx.trace(g.gb, sc.eye, api.trace_out(*whole))
    rows = lambda t, r0, r1: t[r0 * W * 4:r1 * W * 4]  # noqa: E731
    cuts = [0, 1, 17, 49, 273, 1169, 2065, 2961, 3857, H]
    for r0, r1 in zip(cuts, cuts[1:]):
        gb = api.gbuffer(rows(g.gpos, r0, r1), rows(g.gnrm, r0, r1), rows(g.galb, r0, r1), W, r1 - r0)
        ctx.trace(gb, sc.eye, api.trace_out(*(rows(t, r0, r1) for t in bands[:3]), bands[3]))
    torch.cuda.synchronize()
    assert float(whole[0].abs().sum()) > 0
    for a, b in zip(whole, bands):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    ctx.close()
