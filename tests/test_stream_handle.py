"""The stream that calls without one go to: torch's current stream, by its
handle where torch has a call for that (a private one), else by the Stream
object."""

from __future__ import annotations

import types

import pytest
import torch

from vct_gb300 import api


@pytest.mark.parametrize("private,initialised,want", [(True, True, 700 + 3), (False, True, 55), (True, False, 55)])
def test_current_stream(monkeypatch, private, initialised, want):
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: initialised)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=55))
    if private:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 700 + d, raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert api._stream(None) == want
    assert api._stream(9) == 9 and api._stream(types.SimpleNamespace(cuda_stream=8)) == 8
