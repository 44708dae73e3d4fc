"""stream_handle without a GPU: the handle of a given stream, and the current stream's by torch's
raw call or, where a torch lacks it, through the Stream object."""
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from thermal_inflation_phase_transition_b200._common import stream_handle  # noqa: E402


@pytest.mark.parametrize("raw", [True, False])
def test_current(monkeypatch, raw):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=0x20))
    if raw:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 0x10 + d, raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert stream_handle().value == (0x11 if raw else 0x20)


def test_given():
    assert stream_handle(SimpleNamespace(cuda_stream=0x30)).value == 0x30
