"""Switches that choose between ways of the same result."""
import os
import subprocess
import sys

import pytest
import torch

from soap_tp_b200.engine import kernels as k

SIZES = [(8192, 8192, False), (4096, 4096, True), (14336, 4096, False)]


@pytest.fixture
def restored():
    yield
    k.use_cta_pairs(os.environ.get("SOAP_TP_GEMM_CTA_PAIRS", "1") != "0")


@pytest.mark.parametrize("size", SIZES)
def test_products_of_fp16_pairs_honour_the_pair_switch(size, restored):
    k.use_cta_pairs(True)
    assert k._C.half_on_pairs(*size)
    k.use_cta_pairs(False)
    assert not k._C.half_on_pairs(*size)


@pytest.mark.parametrize("shape,small", [((512, 1376), True), ((1, 1), True), ((128, 2048), True), ((2048, 2048), False),
                                         ((8192, 8192), False), ((128, 14336), False), ((14336, 64), False)])
@pytest.mark.parametrize("pairs", [True, False])
def test_which_steps_share_launches_does_not_hang_on_the_pair_switch(shape, small, pairs, restored):
    """Each step of a shared launch has scratch of its own, which large matrices cannot afford."""
    k.use_cta_pairs(pairs)
    assert k._C.steady_step_shares(*shape) is small


def test_the_pair_switch_of_the_environment():
    code = "from soap_tp_b200.engine import kernels as k; print(k._C.half_on_pairs(8192, 8192, False))"
    for value, expected in (("0", "False"), ("1", "True")):
        out = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, SOAP_TP_GEMM_CTA_PAIRS=value), text=True,
                             capture_output=True, check=True)
        assert out.stdout.strip().endswith(expected)


class FakeStream:
    made = 0

    def __init__(self, device=None, priority=0):
        FakeStream.made += 1
        self.priority, self.cuda_stream = priority, 1000 + FakeStream.made


@pytest.fixture
def streams(monkeypatch):
    """Streams of the caller: (handle, priority) becomes current."""
    from soap_tp_b200.engine import local

    current = FakeStream()
    monkeypatch.setattr(torch.cuda, "Stream", FakeStream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: current)
    monkeypatch.setattr(local, "_SIDE_STREAMS", {})

    def side_of(handle, priority=0):
        current.cuda_stream, current.priority = handle, priority
        return local._side_stream(torch.device("cuda", 0), handle)

    return local, side_of


def test_every_callers_stream_has_averages_of_its_own(streams):
    local, side_of = streams
    first, second = side_of(1), side_of(2)
    assert first != second and side_of(1) == first and side_of(2) == second
    assert {first, second}.isdisjoint({1, 2})


def test_averages_have_the_callers_priority(streams):
    local, side_of = streams
    for handle, priority in ((1, 0), (2, -1)):
        handle = side_of(handle, priority)
        stream, = (s for s in local._SIDE_STREAMS.values() if s.cuda_stream == handle)
        assert stream.priority == priority


def test_streams_that_come_and_go_are_not_kept(streams):
    local, side_of = streams
    for handle in range(500):
        side_of(handle)
    assert len(local._SIDE_STREAMS) <= 64


def test_the_overlap_switch_leaves_everything_on_the_callers_stream(streams, monkeypatch):
    local, side_of = streams
    monkeypatch.setattr(local, "OVERLAP_GRAM", False)
    assert side_of(7) == 7 and not local._SIDE_STREAMS
