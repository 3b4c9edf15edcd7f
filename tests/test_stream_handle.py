"""The stream handle that the passes hand to the library, with and without torch's raw-handle call
(which is not of its public interface)."""
from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("raw", [True, False])
def test_current_stream_handle(monkeypatch, raw):
    import torch
    from helio_b200 import passes as P

    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: SimpleNamespace(cuda_stream=71))
    if raw:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 70 + d, raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert P._stream_ptr(None) == (73 if raw else 71)
    assert P._stream_ptr(SimpleNamespace(cuda_stream=5)) == 5
