"""Kernels launched with programmatic dependence, which may start before the
kernel in front of them has ended: alternating chains of them, directly and
captured into a graph, give the bits that each gives by itself."""

from __future__ import annotations

import pytest

from helpers import GpuScene
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def test_alternating_training_steps():
    """Steps of two networks in turn on one stream, one of them started anew
    in between, against each network alone with a wait after every step."""
    import torch

    torch.manual_seed(3)
    rows, targets = torch.randn(4000, 42, device="cuda"), torch.rand(4000, 3, device="cuda")
    sizes = [4000, 129, 1, 2500, 4000, 300] * 5

    def run(nets, wait):
        losses = torch.zeros(2, len(sizes), device="cuda")
        for k, n in enumerate(sizes):
            for i, m in nets:
                if i == 1 and k == 11:
                    m.set_params(start)
                m.train_step(rows[k:], targets[k:], None, n - k if n > k else 1, 1e-3, losses[i, k:])
                if wait:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        return losses, [m.params() for _, m in nets]

    start = api.Mlp(seed=8).params()
    losses, params = run([(0, api.Mlp(seed=6)), (1, api.Mlp(seed=7))], False)
    for i, seed in ((0, 6), (1, 7)):
        alone, p = run([(i, api.Mlp(seed=seed))], True)
        assert torch.equal(alone[i], losses[i])
        assert (p[0] == params[i]).all()


@pytest.mark.parametrize("size", [(61, 35), (1300, 900)])
def test_captured_depth_passes(size):
    import torch

    sc = scenes.cornell(seed=3, dim=16, gbuffer=size)
    g = GpuScene(sc)
    planes = (g.sm, g.gpos, g.gnrm, g.galb)
    want = [t.clone() for t in planes]
    graph, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=st):
        api.render_shadowmap(g.tris, sc, g.sm)
        api.render_gbuffer(g.tris, sc, g.keys, g.gpos, g.gnrm, g.galb)
    for _ in range(3):
        for t in planes:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(planes, want))


@pytest.mark.parametrize("columns", [1, 4], ids=["points", "walk"])
def test_captured_tessellation(columns):
    """Both kernels of the tessellation voxeliser, which start before the kernel
    in front of them has ended, in frames under capture: one of columns of
    slivers, one of boxes, in turn."""
    import torch

    sc = scenes.large_family(3, dim=64, shadow=64, gbuffer=(64, 48), n_boxes=200, n_cyl=columns, cyl_segments=columns * 75)
    g = GpuScene(sc)
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc, voxelize_tesselation=1))
        out = g.new_outputs()

        def frame():
            ctx.frame(g.tris, g.lights, g.shadow, sc.eye, g.gb, api.trace_out(*out))

        frame()
        torch.cuda.synchronize()
        want, stats = [t.clone() for t in out[:3]], ctx.stats()
        graph, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=st):
            frame()
        for _ in range(4):
            for t in out:
                t.zero_()
            graph.replay()
        torch.cuda.synchronize()
        assert float(want[0].abs().sum()) > 0
        assert all(torch.equal(a, b) for a, b in zip(out, want))
        assert ctx.stats() == stats
