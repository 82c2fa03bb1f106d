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


@pytest.mark.parametrize("source,kernel,constants", [("generic_kernels.cu", "rope_kv_write_kernel", {"inv_freq"}),
                                                     ("generic_kernels.cu", "gated_mul_kernel", set()),
                                                     ("generic_kernels.cu", "gated_mul_vec_kernel", set())])
def test_inputs_of_dependent_kernels_with_restricted_outputs(source, kernel, constants):
    """Outputs may be ``__restrict__``, and what no kernel writes; an input that a predecessor writes may not."""
    body = function((CSRC / source).read_text(), kernel)
    assert body.index("sp_wait_for_predecessor();") < body.index("blockIdx")
    assert "__ldg" not in body and ".nc" not in body and "__ldcs" not in body
    parameters = body[:body.index("{")].split(",")
    restricted = [p for p in parameters if "__restrict__" in p]
    assert {p.split()[-1].rstrip(") ") for p in restricted if p.strip().startswith("const")} <= constants
    assert any("const" in p and "__restrict__" not in p for p in parameters)


def test_weights_are_asked_for_ahead_only_behind_an_ordinary_launch():
    """``w_settled`` lets a product read its weight before its predecessor has ended. The first kernel of a step's layers, in
    both runners, is launched in the ordinary way, so all that was on the stream before the step has ended by then."""
    package = CSRC.parent
    assert "norm_prepare_kernel<<<" in (CSRC / "generic_kernels.cu").read_text()
    sets = re.compile(r"w_settled *= *(True|1)\b")
    users = {p.name for p in list(package.rglob("*.py")) + list(CSRC.glob("*.cu*")) if sets.search(p.read_text())}
    assert users == {"fused_prefill.py", "host_step.cu"}
    runner = (package / "engine" / "fused_prefill.py").read_text()
    body = runner[runner.index("    def run(self"):]
    assert body.index("K.norm_prepare(h, self.fields[0]") < body.index("for i, ")
    runner = (CSRC / "host_step.cu").read_text()
    body = runner[runner.index("SP_API int sp_host_step_prompt_layers"):]
    assert body.index("k.norm_prepare(st.h, layers[0].norm1") < body.index("for (int l = 0;")


@pytest.mark.parametrize("source", ["tc_mid.cu", "tc_stream.cu", "tc_gemm.cu"])
def test_epilogue_operands_of_dependent_products(source):
    text = (CSRC / source).read_text()
    for at in re.finditer(r"__ldg\(", text):
        assert any(c in text[at.end():at.end() + 40] for c in CONSTANT), text[at.start():at.end() + 60]
    assert "ld.global.nc" not in text
