"""The Python binding's plumbing (no GPU)."""
import types


def test_current_stream_without_private_torch_names(monkeypatch):
    from excalibur_b200 import capi
    stream = types.SimpleNamespace(cuda_stream=1234)
    public = types.SimpleNamespace(_C=types.SimpleNamespace(), cuda=types.SimpleNamespace(current_stream=lambda: stream))
    monkeypatch.setattr(capi, "_TORCH", public)
    assert capi._stream() == 1234
    asked = []
    public._C._cuda_getDevice = lambda: 3
    public._C._cuda_getCurrentRawStream = lambda device: asked.append(device) or 77
    assert capi._stream() == 77 and asked == [3]
