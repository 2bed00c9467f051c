"""CPU: what the GEMM kernels' epilogue warps may touch and when.  Broken, each of these would be a race that shows on a
device only now and then, so the places and the order are looked up in the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bytetransformer_b200", "csrc")


def _code():
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "gemm_sm100.cu")).read())


def _body(start):
    """The text from `start` (a definition) to the closing brace at the same indentation."""
    src = _code()
    at = src.index(start)
    return src[at:src.index("\n}\n", at)]


@pytest.mark.parametrize("kernel,tile", [("gemm_f16_kernel(const", "BLOCK_N"), ("gemm_f16_pair_kernel(const", "kTileN")])
def test_an_epilogue_warp_keeps_its_bias_where_no_other_warp_writes(kernel, tile):
    """Nothing orders one warp's reads of a tile's bias before another warp's writes of a later tile's: the arrive that
    hands an accumulator back from a pair is relaxed.  So each warp has a slice of its own."""
    body = _body(kernel)
    assert re.findall(r"bias_s = ([^;]*);", body) == [f"bias_slice<{tile}>(bars, e)"]
    assert body.count("bias.put(bias_s, lane);") == 1
    # a warp's reads of one tile are behind a __syncwarp before it writes the next tile's
    tail = body[body.index("bias.put(bias_s, lane);"):]
    assert tail.index("__syncwarp();") < tail.index("mbar_arrive")


@pytest.mark.parametrize("tile", [64, 128, 256])
def test_bias_slices_lie_apart_and_inside(tile):
    code = _code()
    warps = int(re.search(r"constexpr int kEpiWarps = (\d+);", code).group(1))
    size = re.search(r"constexpr int bias_bytes\(int tile_n\) \{ return ([^;]*); \}", code).group(1)
    size = eval(size.replace("/", "//"), {"kEpiWarps": warps, "tile_n": tile})
    offset = re.search(r"kBarBytes\) \+ ([^;]*);", _body("__half* bias_slice(")).group(1).replace("/", "//")
    starts = [2 * eval(offset, {"epi_warp": e, "TILE_N": tile}) for e in range(warps)]  # bytes
    own = tile // 2 * 2  # half of the tile's columns, two bytes each
    assert all(b - a >= own for a, b in zip(starts, starts[1:])) and starts[0] == 0 and starts[-1] + own <= size
    assert all(s % 16 == 0 for s in starts)  # read 16 bytes at a time


@pytest.mark.parametrize("kernel", ["gemm_f16_kernel(const", "ln_gemm_body("])
def test_tensor_memory_goes_early_only_where_no_wait_has_given_up(kernel):
    """The epilogue goes on after a wait that gave up, and MMAs may be in flight then: the MMA warp may free tensor memory
    ahead of the CTA's end only on the answer that every accumulator came back and nobody gave up."""
    body = _body(kernel)
    assert body.split("if (*abort_flag != 0)")[0].count("tmem_dealloc(") == 1
    assert re.search(r"if \(accumulators_back\(acc_empty, tiles, abort_flag, args\.status, kStatusGemmMmaTimeout\)\) \{\s*"
                     r"tc_fence_after\(\);\s*tmem_dealloc\([^;]*\);\s*tmem_freed = true;\s*\}", body)


@pytest.mark.parametrize("kernel", ["gemm_f16_kernel(const", "gemm_f16_ln_kernel(const"])
def test_tensor_memory_is_freed_behind_the_join_otherwise(kernel):
    """Whatever keeps it from being freed early raises the flag, so the other place is behind the flag and the drain."""
    body = _body(kernel)
    end = body[body.rindex("__syncthreads();"):]
    flag, drain = end.index("if (*abort_flag != 0) {"), end.index("__nanosleep(2000)")
    free = end.index("if (warp == 1 && !tmem_freed) {")
    assert flag < drain < free < end.index("tmem_dealloc(")
    assert end.count("\n  }") == 1  # one block, the flag's


@pytest.mark.parametrize("kernel", ["gemm_f16_pair_kernel(const", "gemm_f16_pair_ln_kernel(const"])
def test_a_pair_frees_tensor_memory_behind_its_join(kernel):
    body = _body(kernel)
    assert body.count("tcgen05.dealloc") == 1
    assert body.rindex("cluster_sync_all();") < body.index("tcgen05.dealloc")
