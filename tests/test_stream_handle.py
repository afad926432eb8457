"""The stream handle that the Python entry points pass on, without a GPU."""
import types

import pytest

torch = pytest.importorskip("torch")


@pytest.fixture
def fake(monkeypatch):
    """A torch whose current stream is 77, by the public call and by the raw one."""
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=77))
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 70 + d, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 7, raising=False)
    return monkeypatch


def test_raw_handle(vsc, fake):
    fake.setattr(torch.cuda, "current_stream", lambda *a: pytest.fail("not needed"))
    assert vsc._stream().value == 77


@pytest.mark.parametrize("missing", ["_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_public_call_where_torch_lacks_the_raw_one(vsc, fake, missing):
    fake.delattr(torch._C, missing)
    assert vsc._stream().value == 77


def test_given_stream(vsc, fake):
    assert vsc._stream(types.SimpleNamespace(cuda_stream=5)).value == 5
