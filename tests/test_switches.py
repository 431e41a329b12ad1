"""Switches that choose between ways of the same result."""
import os
import subprocess
import sys

import pytest

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


def test_the_pair_switch_of_the_environment():
    code = "from soap_tp_b200.engine import kernels as k; print(k._C.half_on_pairs(8192, 8192, False))"
    for value, expected in (("0", "False"), ("1", "True")):
        out = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, SOAP_TP_GEMM_CTA_PAIRS=value), text=True,
                             capture_output=True, check=True)
        assert out.stdout.strip().endswith(expected)
