"""The current stream's handle, with and without torch's function for raw
handles, which is not public."""
import pytest

from einspline_gb300 import api


@pytest.mark.parametrize("has_raw", [True, False])
def test_handle_of_the_current_stream(monkeypatch, has_raw):
    torch = pytest.importorskip("torch")
    for name in ("_cuda_getCurrentRawStream", "_cuda_getDevice"):
        monkeypatch.delattr(torch._C, name, raising=False)
    if has_raw:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 40 + device, raising=False)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 2)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: type("S", (), {"cuda_stream": 42}))
    assert api._stream(torch, None) == 42
    assert api._stream(torch, type("S", (), {"cuda_stream": 7})) == 7
