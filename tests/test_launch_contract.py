"""CPU: what the kernels of a call may take for granted when they start ahead of their predecessor's end (the rules stand
in csrc/common.cuh).  Broken, each would be a race that shows on a device only now and then, so the order of the two
instructions and the plain first launch are looked up in the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bytetransformer_b200", "csrc")


def _body(name, start):
    """The text from `start` (a definition) to the closing brace at the same indentation."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    at = src.index(start)
    return src[at:src.index("\n}\n", at)]


@pytest.mark.parametrize("name,kernel", [("offsets.cu", "pack_rows_kernel("), ("offsets.cu", "mask_bits_kernel("),
                                         ("embed_pool.cu", "embedding_layernorm_kernel(")])
def test_second_kernels_of_a_call_trigger_after_their_own_wait(name, kernel):
    body = _body(name, kernel)
    assert body.index("pdl_wait();") < body.index("pdl_launch_dependents();")
    assert "return" not in body[:body.index("pdl_launch_dependents();")]


@pytest.mark.parametrize("entry,first", [
    ("static int stack_padded(", "launch_build_offsets("), ("static int stack_general(", "launch_uniform_offsets("),
    ("int bt_stack_forward_packed(", "run_layer("), ("int bt_gemm(", "run_gemm("), ("int bt_gemm_layernorm(", "run_gemm("),
    ("int bt_add_bias_residual_layernorm(", "launch_layernorm("),
    ("int bt_add_bias_residual_layernorm_restore(", "launch_layernorm_restore("),
])
def test_first_kernel_of_a_call_that_reads_parameters_early_is_launched_plainly(entry, first):
    body = _body("encoder.cu", entry)
    assert body.index("pdl_next_launch_plain();") < body.index(first)


def test_offsets_are_read_early_only_inside_a_forward():
    src = open(os.path.join(CSRC, "encoder.cu")).read()
    calls = re.findall(r"run_mha\(h,[^;]*?, (true|false)(?:, gm)?\)", src)
    assert sorted(calls) == ["false", "true"]  # bt_attention and run_layer
