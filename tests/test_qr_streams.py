"""The streams of the factorisations and how they are joined, with CUDA's objects recorded instead of made."""
import pytest
import torch

from soap_tp_b200.engine import qr


class Stream:
    def __init__(self, device=None, priority=0):
        self.priority, self.waited = priority, []

    def wait_event(self, event):
        self.waited.append(event)


class Event:
    def record(self, stream=None):
        self.stream = stream


@pytest.fixture
def main(monkeypatch):
    """The caller's stream."""
    stream = Stream()
    monkeypatch.setattr(torch.cuda, "Stream", Stream)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stream)
    for streams in ("_PANEL_STREAMS", "_SIDE_STREAMS"):
        monkeypatch.setattr(qr, streams, {})
    return stream


@pytest.mark.parametrize("slot", [0, 1])
def test_the_accumulation_of_q_goes_before_nobody(main, slot):
    """A lone factorisation's trailing updates run on the caller's stream, and its next panel waits for them."""
    accumulation, panels = qr._q_stream(main, slot), qr._panel_stream(main, slot)
    assert accumulation.priority >= main.priority > panels.priority      # (lower numbers go first)
    assert accumulation is qr._q_stream(main, slot) and accumulation is not panels
