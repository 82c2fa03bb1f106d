"""Kernels that may be resident before their predecessor ends read what it writes by ordinary loads behind the wait: neither a
read-only load nor a ``const __restrict__`` parameter, from which the compiler may make one, will do. Held by the source."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "spissa_b200" / "csrc"
# what no kernel writes: weights
CONSTANT = ("ep.next_w",)


def function(text: str, name: str) -> str:
    """The kernel ``name`` of a source: its parameters and its body."""
    start = re.search(r"__global__[^;{]*\b" + name + r"\(", text).end()
    depth, at = 0, text.index("{", start)
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError(f"{name} has no end")


@pytest.mark.parametrize("source,kernel", [("generic_kernels.cu", "gemm_stream_f32_kernel"),
                                           ("generic_kernels.cu", "attention_decode_f32_kernel"), ("gemv_kernels.cu", "gemv_kernel")])
def test_parameters_and_loads_of_a_dependent_kernel(source, kernel):
    text = (CSRC / source).read_text()
    body = function(text, kernel)
    assert "sp_wait_for_predecessor();" in body
    assert "__restrict__" not in body and "__ldg" not in body and ".nc" not in body and "__ldcs" not in body


@pytest.mark.parametrize("source", ["tc_mid.cu", "tc_stream.cu", "tc_gemm.cu"])
def test_epilogue_operands_of_dependent_products(source):
    text = (CSRC / source).read_text()
    for at in re.finditer(r"__ldg\(", text):
        assert any(c in text[at.end():at.end() + 40] for c in CONSTANT), text[at.start():at.end() + 60]
    assert "ld.global.nc" not in text
