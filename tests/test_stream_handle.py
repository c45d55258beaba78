"""The stream handle of a call (CPU): the caller's stream, else torch's current one, by the raw
call where torch has it and by the Stream object where it does not."""
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from l3es import _native  # noqa: E402


def test_handle_of_the_given_and_of_the_current_stream(monkeypatch):
    assert _native._stream(SimpleNamespace(cuda_stream=5)) == 5
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 2)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: SimpleNamespace(cuda_stream=7))
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 100 + d, raising=False)
    assert _native._stream() == 102
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    assert _native._stream() == 7
