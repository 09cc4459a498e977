"""The calls' stream lookup: torch's raw-stream function where this torch has it, else the public one."""
import types

import torch

from gbblas import api


def test_falls_back_to_the_public_lookup(monkeypatch):
    t = types.SimpleNamespace(device="cuda:1", get_device=lambda: 1)
    monkeypatch.setattr(api, "_raw_stream", lambda index: 100 + index)
    assert api._stream_of(t) == 101
    monkeypatch.setattr(api, "_raw_stream", None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device: types.SimpleNamespace(cuda_stream=(7, device)))
    assert api._stream_of(t) == (7, "cuda:1")
