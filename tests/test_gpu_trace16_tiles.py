"""The 16-cone trace by halves of tiles, at images that end inside a half: the
whole image against the oracle, the listed tiles against the whole image; and
an image of a few tiles to an SM takes its share of a large one's time."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from helpers import GpuScene, read_chain
from vct_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (16, 8), (17, 9), (15, 16), (33, 40), (130, 71)])
def test_odd_images(size):
    import torch

    W, H = size
    sc = scenes.cornell(seed=6, dim=32, gbuffer=size)
    g = GpuScene(sc)
    _, gbuf = g.host_inputs()
    with api.Context(api.config_for(sc)) as ctx:
        ctx.set_params(api.scene_params(sc))
        ctx.frame_volume(g.tris, g.lights, g.shadow, sc.eye)
        ref, out = torch.full((W * H * 4,), -1.0, device="cuda"), torch.full((W * H * 4,), -1.0, device="cuda")
        api.trace_reference16(ctx, g.gb, sc.eye, ref)
        stats = api.learned_trace(ctx, api.Mlp(seed=4), g.gb, sc.eye, out, 1e-6, want_stats=True)
        chain = read_chain(ctx)
    got = ref.cpu().numpy().reshape(-1, 4)
    want, _ = O.trace_reference16(sc, chain, gbuf[0], gbuf[1], np.arange(W * H, dtype=np.int32), precision=32, nthreads=8)
    assert np.linalg.norm(got[:, :3] - want[:, :3]) <= 1e-4 * max(np.linalg.norm(want[:, :3]), 1e-30)
    assert np.all(got[:, 3] == 0.0)
    # an untrained network: every tile with a covered probe in the image is listed, and holds the trace
    cov = gbuf[0].reshape(H, W, 4)[..., 3] != 0
    r, o = ref.view(H, W, 4).cpu().numpy(), out.view(H, W, 4).cpu().numpy()
    listed = 0
    for y in range(0, H, 16):
        for x in range(0, W, 16):
            probes = [cov[y + a, x + b] for a in (4, 12) for b in (4, 12) if y + a < H and x + b < W]
            if any(probes) and np.any(r[y:y + 16, x:x + 16]):
                listed += 1
                assert np.array_equal(o[y:y + 16, x:x + 16, :3], r[y:y + 16, x:x + 16, :3])
    assert stats["fallback_tiles"] >= listed


def test_mid_size_images_take_their_share():
    """800 x 450 pixels are 0.39 of 1280 x 720: some 0.48 of the time, and 0.59
    where a few SMs end a heavy tile behind the others."""
    import torch

    def best(size):
        sc = scenes.cornell(seed=1, dim=128, gbuffer=size)
        g = GpuScene(sc)
        with api.Context(api.config_for(sc)) as ctx:
            ctx.set_params(api.scene_params(sc))
            ctx.frame_volume(g.tris, g.lights, g.shadow, sc.eye)
            ref, times = torch.zeros(size[0] * size[1] * 4, device="cuda"), []
            for _ in range(6):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for _ in range(8):
                    api.trace_reference16(ctx, g.gb, sc.eye, ref)
                b.record()
                torch.cuda.synchronize()
                times.append(a.elapsed_time(b))
        return min(times[1:])

    assert best((800, 450)) < 0.54 * best((1280, 720))
