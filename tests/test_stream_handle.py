"""The current stream's handle, with and without torch's private names (no GPU)."""
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")
import ugemm_gb300 as ug  # noqa: E402


def test_stream_handle_without_private_names(monkeypatch):
    monkeypatch.setattr(ug, "_raw_stream", None)
    monkeypatch.setattr(torch.cuda, "init", lambda: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=7))
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert ug._stream_ptr(None) == 7
    assert ug._stream_ptr(SimpleNamespace(cuda_stream=9)) == 9
