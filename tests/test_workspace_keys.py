"""Scratch planes are shared by shape and by nothing else: planes of another form are other planes."""
import torch

from soap_tp_b200.engine import kernels as k
from soap_tp_b200.engine import local


def test_planes_of_another_form_are_other_planes(monkeypatch):
    monkeypatch.setattr(local, "_WORKSPACES", {})
    device = torch.device("cpu")
    get = lambda **form: local.workspace_planes("X", 64, 32, device, **form)
    monkeypatch.setattr(k, "MIXED_CORRECTIONS", True)
    vector, block, one = get(), get(blocked=True), get(terms=1)
    assert not vector.blocked and block.blocked and one.terms == 1 and vector.terms == 2
    assert vector.largest is not None and block.scale.shape == (1, 32)
    assert get() is vector and get(blocked=True) is block and get(terms=1) is one
    monkeypatch.setattr(k, "MIXED_CORRECTIONS", False)
    assert isinstance(get(), k.Planes)
