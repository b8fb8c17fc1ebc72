"""Host-side Python that needs no GPU."""

import types

import pytest
import torch

from dromos_b200 import host


@pytest.mark.parametrize("short_way", [True, False])
def test_current_stream_with_and_without_torchs_short_way(monkeypatch, short_way):
    monkeypatch.setattr(host, "_raw_stream_of_device", (lambda device: 1000 + device) if short_way else None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=1003))
    assert host._raw_stream() == 1003
