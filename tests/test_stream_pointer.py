"""The stream handle the calls take: an explicit stream's, else the current one's, with and without
torch's unpublished call for it (CPU: fakes of torch's calls)."""
import types

import pytest


@pytest.mark.parametrize("published_only", [False, True])
def test_stream_pointer(monkeypatch, published_only):
    torch = pytest.importorskip("torch")
    import gbmv
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=77))
    if published_only:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    else:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 74 + device,
                            raising=False)
    assert gbmv._stream_ptr(None) == 77
    assert gbmv._stream_ptr(types.SimpleNamespace(cuda_stream=5)) == 5
