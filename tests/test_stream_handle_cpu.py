"""The stream handle of the functional calls without the private interface of torch that they use where it exists."""
import importlib

import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name", ["_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_stream_without_private_interface(monkeypatch, name):
    from cunn_b200 import functional
    with monkeypatch.context() as m:
        m.delattr(torch._C, name, raising=False)
        m.setattr(torch.cuda, "current_stream", lambda *a: type("S", (), {"cuda_stream": 71})())
        importlib.reload(functional)
        assert functional._stream() == 71
    importlib.reload(functional)
