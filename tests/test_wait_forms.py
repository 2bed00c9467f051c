"""CPU: the roles of the GEMM and attention kernels wait warp by warp.  A wait answers for one lane; where it gives up,
lanes that disagree must not go separate ways into warp-wide instructions, so the kernels use the forms that vote (or,
in a K loop, remember and vote after the loop)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bytetransformer_b200", "csrc")


def _code(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", src)


@pytest.mark.parametrize("name", ["gemm_sm100.cu", "mha_sm100.cu", "embed_pool.cu", "offsets.cu", "encoder.cu"])
def test_kernels_use_the_voting_waits(name):
    assert "mbar_wait_bounded" not in _code(name)


def test_every_latched_loop_ends_in_a_vote():
    code = _code("gemm_sm100.cu")
    loops = [m.end() for m in re.finditer(r"ok = mbar_wait_latched\(ok,", code)]
    assert len(loops) == 4
    for pos in loops:
        commit = code.index("umma_commit", pos)
        assert "ok = __all_sync(0xffffffffu, ok) != 0;" in code[pos:commit]
