"""CPU: what the kernels of a call may take for granted when they start ahead of their predecessor's end.  Kernels that
read parameters ahead of their dependency wait rely on the call's first kernel being launched the ordinary way; forgotten,
it would be a race that shows on a device only now and then, so it is looked up in the source."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bytetransformer_b200", "csrc")


def _body(name, start):
    """The text from `start` (a definition) to the closing brace at the same indentation."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    at = src.index(start)
    return src[at:src.index("\n}\n", at)]


@pytest.mark.parametrize("entry,first", [
    ("static int stack_padded(", "launch_build_offsets("), ("static int stack_general(", "launch_uniform_offsets("),
    ("int bt_stack_forward_packed(", "run_layer("), ("int bt_gemm(", "run_gemm("), ("int bt_gemm_layernorm(", "run_gemm("),
    ("int bt_add_bias_residual_layernorm(", "launch_layernorm("),
    ("int bt_add_bias_residual_layernorm_restore(", "launch_layernorm_restore("),
])
def test_first_kernel_of_a_call_that_reads_parameters_early_is_launched_plainly(entry, first):
    body = _body("encoder.cu", entry)
    assert body.index("pdl_next_launch_plain();") < body.index(first)
