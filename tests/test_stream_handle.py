"""The current stream's handle without torch's private entry (no GPU)."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from planet_renderer_gb300 import _native


@pytest.fixture
def fake_cuda(monkeypatch):
    """Stands in for a CUDA device: device 3's current stream is 0x300."""

    monkeypatch.setattr(torch.cuda, "init", lambda: None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda index: SimpleNamespace(cuda_stream=0x100 * index))
    monkeypatch.setattr(_native, "_current_raw_stream", None)


def test_public_stream_where_the_private_entry_is_missing(fake_cuda, monkeypatch):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert _native.stream(torch.device("cuda", 3)).value == 0x300
    assert _native.stream(torch.device("cuda")).value == 0x300
    with pytest.raises(ValueError):
        _native.stream(torch.device("cpu"))


def test_private_entry_where_it_is_there(fake_cuda, monkeypatch):
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 0x1000 + index, raising=False)
    assert _native.stream(torch.device("cuda", 3)).value == 0x1003
