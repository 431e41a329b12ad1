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


@pytest.mark.parametrize("fails", ["beside", "panel"])
def test_what_was_issued_before_a_failure_is_waited_for(main, monkeypatch, fails):
    """Out of memory beside the factorisations: they still read the orders of their columns, whose memory the caller's stream is
    given next."""
    import contextlib

    working = []

    def steps(matrix, Q, order, slot, readers=None):
        working.extend(stream for stream in (current[-1], qr._panel_stream(matrix.device, slot)) if stream not in working)
        yield
        if fails == "panel" and slot == 1:
            raise torch.OutOfMemoryError("out of memory")
        yield

    @contextlib.contextmanager
    def on(stream):
        current.append(stream)
        yield
        current.pop()

    def beside():
        if fails == "beside":
            raise torch.OutOfMemoryError("out of memory")

    current = [main]
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(qr, "_factorisation_steps", steps)
    jobs = [(torch.zeros(4, 4), torch.zeros(4, 4), torch.arange(4)) for _ in range(2)]
    with pytest.raises(torch.OutOfMemoryError):
        qr.householder_qr_pair(jobs, beside)
    assert len(working) == 4 and main not in working
    assert {id(event.stream) for event in main.waited} >= {id(stream) for stream in working}
