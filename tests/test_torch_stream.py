"""The handle of torch's current stream, from a torch with and without the private
calls that are the short way to it (no GPU: torch's CUDA calls are stood in for)."""
import pytest

import recon_gb300 as rg

torch = pytest.importorskip("torch")


class Stream:
    cuda_stream = 77


@pytest.mark.parametrize("missing", ["", "_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_current_stream_handle(monkeypatch, missing):
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream())
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 3, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 70 + device, raising=False)
    if missing:
        monkeypatch.delattr(torch._C, missing)
    assert rg._torch_stream() == (77 if missing else 73)
