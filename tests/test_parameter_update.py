"""Which tensors the one-pass parameter updates take by address; the others are left to the tensor operations."""
import pytest
import torch

from soap_tp_b200.engine import kernels as k


class Wrapped(torch.Tensor):
    """A subclass without storage of its own, as distributed and quantised parameters are."""

    @staticmethod
    def __new__(cls, inner):
        return torch.Tensor._make_wrapper_subclass(cls, inner.shape, dtype=inner.dtype, device=inner.device)

    def __init__(self, inner):
        self.inner = inner

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise NotImplementedError


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *arguments: self.calls.append(name)


@pytest.fixture
def launches(monkeypatch):
    recorder = Recorder()
    monkeypatch.setattr(k, "_C", recorder)
    monkeypatch.setattr(k, "_stream", lambda: 0)
    return recorder.calls


@pytest.mark.parametrize("wrap", [lambda t: t, Wrapped, lambda t: t.to("meta")])
def test_tensors_that_are_not_plain_memory_of_the_current_device_are_refused(launches, wrap):
    p, other = wrap(torch.zeros(8)), [wrap(torch.zeros(8)) for _ in range(3)]
    assert not k.apply_update(p, other[0], 1.0, 0.1)
    assert not k.adamw_update(p, *other, 0.9, 0.95, 0.1, 0.05, 1e-8, 1.0, 0.1)
    assert launches == []


def test_one_subclass_among_plain_tensors_is_enough(launches):
    assert not k._addressable(torch.zeros(8), Wrapped(torch.zeros(8)))


class OnDevice:
    """Stands for a plain tensor on a GPU."""

    dtype, shape, layout = torch.float32, torch.Size([8]), torch.strided

    is_cuda = True

    def __init__(self, index):
        self.index = index

    def get_device(self):
        return self.index

    def is_contiguous(self):
        return True

    def is_neg(self):
        return False


@pytest.mark.parametrize("indices,taken", [((0, 0), True), ((1, 1), False), ((0, 1), False), ((1, 0), False)])
def test_only_tensors_of_the_current_device_are_taken(monkeypatch, indices, taken):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(k, "_PLAIN_TENSORS", (OnDevice,))
    assert k._addressable(*(OnDevice(i) for i in indices)) is taken
