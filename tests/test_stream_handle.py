"""The stream of a call without one: torch's current stream, also where torch does not offer its raw
handle (CPU: torch's side is replaced)."""
import types

import pytest

torch = pytest.importorskip("torch")


@pytest.fixture()
def current(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=1234))
    return monkeypatch


@pytest.mark.parametrize("missing", ["_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_without_the_raw_handle(current, missing):
    import cuyashe_gb300

    current.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 99, raising=False)
    current.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    assert cuyashe_gb300._stream_handle(None) == 99
    current.delattr(torch._C, missing)
    assert cuyashe_gb300._stream_handle(None) == 1234


def test_before_cuda_is_initialised(current):
    import cuyashe_gb300

    current.setattr(torch.cuda, "is_initialized", lambda: False)
    assert cuyashe_gb300._stream_handle(None) == 1234


def test_given_streams():
    import cuyashe_gb300

    assert cuyashe_gb300._stream_handle(7) == 7
    assert cuyashe_gb300._stream_handle(types.SimpleNamespace(cuda_stream=8)) == 8
