"""The cone tracer's two kernels (a warp to 32 pixels; four, for launches of
few pixels) give the same bits for every sampler and kind of march: an image
of 2,640 tiles, which takes the first, against its bands, which take the second
(the last one the first again, for some).  And the line between them is where
neither costs much."""

from __future__ import annotations

import pytest

from helpers import GpuScene
from vct_gb300 import _lib as L
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu

FILTERS = dict(software=L.VCT_FILTER_SOFTWARE, hybrid=L.VCT_FILTER_HYBRID, texture=L.VCT_FILTER_HARDWARE,
               texture_levels=L.VCT_FILTER_HARDWARE_LEVELS)
MARCHES = dict(plain=(L.VCT_WARP_NONE, 0), map=(L.VCT_WARP_TEXTURE, 0), analytic=(L.VCT_WARP_ANALYTIC, 0),
               perspective=(L.VCT_WARP_PERSPECTIVE, 0), steps_65=(L.VCT_WARP_NONE, 65), map_65=(L.VCT_WARP_TEXTURE, 65))


@pytest.mark.parametrize("march", MARCHES)
@pytest.mark.parametrize("filt", FILTERS)
def test_bands_give_the_whole_images_bits(filt, march):
    import torch

    warp, steps = MARCHES[march]
    W, H = 317, 2100
    sc = scenes.cornell(seed=4, gbuffer=(W, H))
    if steps:
        sc.cone = dict(diffuse=(steps, 0.04, 1.0, 1.0, 0.5), specular=(steps, 0.05, 1.7, 0.5, 0.1))
    g = GpuScene(sc)
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc, trace_filter=FILTERS[filt], warp_mode=warp))
        ctx.frame_volume(g.tris, g.lights, g.shadow, sc.eye)
        whole, bands = g.new_outputs(), g.new_outputs()
        ctx.trace(g.gb, sc.eye, api.trace_out(*whole))
        rows = lambda t, r0, r1: t[r0 * W * 4:r1 * W * 4]  # noqa: E731
        cuts = [0, 1, 18, 146, 585, 1070, H]
        for r0, r1 in zip(cuts, cuts[1:]):
            gb = api.gbuffer(rows(g.gpos, r0, r1), rows(g.gnrm, r0, r1), rows(g.galb, r0, r1), W, r1 - r0)
            ctx.trace(gb, sc.eye, api.trace_out(*(rows(t, r0, r1) for t in bands[:3]), bands[3]))
        torch.cuda.synchronize()
    assert float(whole[0].abs().sum()) > 0
    for a, b in zip(whole, bands):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("warp", [L.VCT_WARP_ANALYTIC, L.VCT_WARP_PERSPECTIVE], ids=["analytic", "perspective"])
@pytest.mark.parametrize("filt", ["texture", "texture_levels"])
def test_few_pixels_do_not_cost_more_than_many(filt, warp):
    """1,200 tiles (307,200 pixels) take about as long as 1,250 (320,000); with
    four warps to 32 pixels, which texture samples do not pay for at that
    size, up to 1.4 times as long."""
    import torch

    def best(size):
        sc = scenes.large_family(1, dim=32, shadow=512, gbuffer=size, n_boxes=1000, n_cyl=8, cyl_segments=64)
        g = GpuScene(sc)
        with api.Context(api.config_for(sc)) as ctx:
            ctx.set_params(api.scene_params(sc, trace_filter=FILTERS[filt], warp_mode=warp))
            ctx.frame_volume(g.tris, g.lights, g.shadow, sc.eye)
            out = g.new_outputs()
            to, times = api.trace_out(*out), []
            for _ in range(8):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for _ in range(20):
                    ctx.trace(g.gb, sc.eye, to)
                b.record()
                torch.cuda.synchronize()
                times.append(a.elapsed_time(b))
        return min(times[1:])

    assert best((640, 480)) < 1.25 * best((800, 400))
