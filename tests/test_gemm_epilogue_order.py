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
