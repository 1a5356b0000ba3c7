"""The default stream of a call: torch's current one once CUDA is in use there,
also where torch has no short way to its handle. No GPU needed."""
import sys
import types

from fgf_b200 import ops


def _torch(initialized, short):
    t = types.ModuleType("torch")
    t.cuda = types.SimpleNamespace(is_initialized=lambda: initialized,
                                   current_stream=lambda: types.SimpleNamespace(cuda_stream=0x1234))
    t._C = types.SimpleNamespace()
    if short:
        t._C._cuda_getDevice = lambda: 3
        t._C._cuda_getCurrentRawStream = lambda device: 0x5000 + device
    return t


def test_without_torch_the_default_stream(monkeypatch):
    monkeypatch.delitem(sys.modules, "torch", raising=False)
    assert ops._stream(None) == 0


def test_current_stream_by_either_way(monkeypatch):
    monkeypatch.setitem(sys.modules, "torch", _torch(True, True))
    assert ops._stream(None) == 0x5003
    monkeypatch.setitem(sys.modules, "torch", _torch(True, False))
    assert ops._stream(None) == 0x1234


def test_default_stream_before_cuda_is_in_use(monkeypatch):
    for short in (True, False):
        monkeypatch.setitem(sys.modules, "torch", _torch(False, short))
        assert ops._stream(None) == 0
