"""Training passes in which a CTA takes more than one tile of 128 rows (their
gradients add up in tensor memory, and every operand tile is overwritten): one
row in the second round, a few, and several rounds with a last partial tile.
Bounds as for the smaller passes."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp as OM
from test_gpu_mlp import _net, _rel, _rows

pytestmark = pytest.mark.gpu


def _sizes():
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return dict(one=128 * sms, one_row_more=128 * sms + 1, two=2 * 128 * sms - 5, three=2 * 128 * sms + 1277)


@pytest.mark.parametrize("size", ["one", "one_row_more", "two", "three"])
def test_gradients_over_several_tiles(size):
    import torch

    n = _sizes()[size]
    m, p = _net()
    x, y, dx, dy = _rows(n, seed=1)
    y[-1], dy[-1] = 100.0, 100.0  # the last row's error is a good part of all
    grad, loss = torch.empty(OM.NPARAMS, device="cuda"), torch.empty(1, device="cuda")
    m.gradients(dx, dy, grad, loss)
    g = grad.cpu().numpy().astype(np.float64)
    _, l_emu, g_emu = OM.forward_backward(p, x, y, emulate_bf16=True)
    assert abs(float(loss.item()) - l_emu) <= 1e-3 * l_emu
    assert _rel(g, g_emu) < 1e-2, _rel(g, g_emu)
    for o, k in ((0, 2688), (2688, 64), (2752, 4096), (6848, 64), (6912, 4096), (11008, 64), (11072, 256), (11328, 4)):
        assert _rel(g[o:o + k], g_emu[o:o + k]) < 2e-2


def test_step_over_listed_rows_of_several_tiles():
    import torch

    n = _sizes()["three"]
    m, p = _net(5)
    _, _, dx, dy = _rows(n, seed=2)
    order = torch.from_numpy(np.random.default_rng(3).permutation(n).astype(np.int32)).cuda()
    grad, loss = torch.empty(OM.NPARAMS, device="cuda"), torch.zeros(2, device="cuda")
    m.gradients(dx[order.long()].contiguous(), dy[order.long()].contiguous(), grad, loss)
    m.train_step(dx, dy, order, n, 1e-3, loss[1:])
    after = m.params().astype(np.float64)
    ref, _, _ = OM.adam(p, grad.cpu().numpy().astype(np.float64), np.zeros_like(p), np.zeros_like(p), 1, 1e-3)
    assert float(loss[0]) == float(loss[1])
    assert np.abs(after - ref).max() < 1e-6
