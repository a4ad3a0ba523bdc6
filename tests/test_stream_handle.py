"""The current stream's handle, with and without torch's raw accessor."""
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")


def test_handle_without_the_raw_accessor(monkeypatch):
    from lumen_b200 import render
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device: SimpleNamespace(cuda_stream=77))
    monkeypatch.setattr(render, "_raw_stream", None, raising=False)
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert render._stream_handle(torch.device("cuda", 0)) == 77


def test_raw_accessor_is_used(monkeypatch):
    from lumen_b200 import render
    monkeypatch.setattr(render, "_raw_stream", lambda index: 1000 + index)
    assert render._stream_handle(torch.device("cuda", 3)) == 1003
