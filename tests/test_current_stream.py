"""The stream that a call from Python is put on: torch's current one, by its public call where the shorter one does not exist."""
from types import SimpleNamespace

import pytest

from tile_fusion_b200 import api


@pytest.mark.parametrize("entry", [True, False])
@pytest.mark.parametrize("initialized", [True, False])
def test_fallback(monkeypatch, entry, initialized):
    cuda = SimpleNamespace(is_initialized=lambda: initialized, current_device=lambda: 3, current_stream=lambda: SimpleNamespace(cuda_stream=77))
    c = SimpleNamespace(_cuda_getCurrentRawStream=lambda device: 100 + device) if entry else SimpleNamespace()
    monkeypatch.setattr(api, "_torch", SimpleNamespace(cuda=cuda, _C=c))
    assert api._stream_ptr() == (103 if entry and initialized else 77)


@pytest.mark.gpu
def test_current_stream(built_lib):
    import torch
    for s in (torch.cuda.default_stream(), torch.cuda.Stream(), torch.cuda.Stream(priority=-1)):
        with torch.cuda.stream(s):
            assert api._stream_ptr() == torch.cuda.current_stream().cuda_stream == s.cuda_stream
