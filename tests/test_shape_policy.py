"""Host-side shape policies of the GEMM launcher (no device needed): the tile width of the one-CTA
kernel, the number of K ranges of the fp32-sum GEMMs that feed a LayerNorm, and when the SM-pair
kernel takes over.  The expected values restate the rules in words; the numbers are for 148 SMs."""
import ctypes as C

import pytest

SMS = 148


@pytest.fixture(scope="module")
def policy():
    from bytetransformer_b200 import _abi, build
    build.build_core()  # no-op when the library is up to date
    lib = _abi.load()
    fn = lib.bt_debug_policy
    fn.restype = C.c_int
    fn.argtypes = [C.c_int] * 5
    return fn


@pytest.mark.parametrize("rows,N,want", [
    (64, 2304, 64),      # never 148 tiles: the narrowest width spreads the weights over most SMs
    (4096, 768, 128),    # 32 row tiles x 3 = 96 tiles of 256 columns, 192 of 128: the widest that fills the SMs
    (18944, 3072, 256),
    (2560, 3072, 256),   # 20 x 12 = 240 tiles
    (128, 192, 64),      # 192 % 128 != 0
])
def test_tile_width_is_the_widest_that_gives_every_sm_a_tile(policy, rows, N, want):
    assert policy(0, rows, N, 768, SMS) == want


@pytest.mark.parametrize("rows,N,K,want", [
    (1536, 768, 3072, 64),   # 12 row tiles: 144 tiles of 64 columns, one wave
    (1537, 768, 3072, 128),  # 13: 156 would be a second wave, 78 of 128 columns are one
    (3072, 768, 3072, 128), (3073, 768, 3072, 128),  # 24: 144 tiles of 128; 25: 150, the plain rule again
    (1537, 768, 768, 64),    # a short K: the second wave is cheap
    (2304, 512, 2048, 64), (2305, 512, 2048, 128),
    (1280, 1024, 4096, 128), (1152, 1024, 4096, 64),
    (1601, 704, 3072, 64), (1793, 704, 3072, 64),    # 704 % 128 != 0
])
def test_a_long_k_takes_wide_tiles_instead_of_a_second_wave_where_all_rows_are_valid(policy, rows, N, K, want):
    assert policy(5, rows, N, K, SMS) == want
    if (rows, want) != (3073, 128):
        assert policy(0, rows, N, K, SMS) == 64   # padded rows may make no tiles


@pytest.mark.parametrize("rows,K,want", [
    (38, 3072, 8), (256, 3072, 8),        # 12 or 24 tiles of 64 columns: 8 ranges still fit 1.5 x the SMs
    (384, 3072, 4), (512, 3072, 4),
    (640, 3072, 2), (1024, 3072, 2),
    (1280, 3072, 1),                      # 120 tiles: even two ranges would be more than 1.5 x the SMs
    (38, 768, 4),                         # 12 K blocks: 8 does not divide them, 4 leaves three blocks per range
    (512, 768, 4), (640, 768, 2),
    (38, 128, 1),                         # two K blocks: nothing to cut
])
def test_k_is_cut_into_as_many_ranges_as_still_fit_the_machine(policy, rows, K, want):
    assert policy(1, rows, 768, K, SMS) == want


@pytest.mark.parametrize("rows,N,want", [
    (18944, 2304, 1), (4352, 2304, 1),    # 17 x 9 = 153 pair tiles >= 148
    (4096, 2304, 0),                      # 16 x 9 = 144
    (18944, 2240, 0),                     # N % 256 != 0
])
def test_pair_kernel_takes_over_at_two_tiles_per_sm_pair(policy, rows, N, want):
    assert policy(2, rows, N, 768, SMS) == want


@pytest.mark.parametrize("rows,hidden,parts,inside,alone", [
    (1, 768, 8, 1, 1), (1024, 768, 2, 1, 1),              # partial sums: one row per CTA
    (399, 768, 1, 1, 1), (400, 768, 1, 4, 4), (512, 256, 1, 1, 1), (513, 256, 1, 1, 0), (1024, 448, 1, 1, 0),
    (1536, 512, 1, 2, 2), (1537, 512, 1, 4, 4), (1536, 640, 1, 4, 4), (2048, 768, 1, 4, 4), (2049, 768, 1, 4, 0), (4096, 1024, 1, 4, 0), (4096, 512, 1, 4, 0),
    (1025, 256, 1, 2, 0), (4096, 448, 1, 2, 0), (1025, 192, 1, 0, 0),
    (4097, 768, 1, 0, 0), (100, 1032, 1, 0, 0),
])
def test_rows_that_share_a_layernorm_cta(policy, rows, hidden, parts, inside, alone):
    assert policy(3, rows, hidden, parts, SMS) == inside
    assert policy(4, rows, hidden, parts, SMS) == alone


@pytest.mark.parametrize("tiles,hidden,all_rows,padded", [
    (31, 768, 0, 0), (32, 768, 1, 0), (39, 768, 1, 0), (40, 768, 1, 1),
    (31, 1024, 0, 0), (32, 1024, 1, 0), (36, 1024, 1, 0), (37, 1024, 0, 0), (38, 1024, 1, 0), (40, 1024, 1, 1),
    (37, 512, 0, 0), (38, 512, 1, 0), (40, 512, 1, 1),   # 74 CTAs are half of the SMs
    (32, 256, 0, 0), (39, 256, 0, 0), (40, 256, 1, 1),
    (64, 320, 0, 0), (64, 1280, 0, 0),                   # widths without the fused kernels
])
def test_layernorm_inside_the_gemm(policy, tiles, hidden, all_rows, padded):
    from bytetransformer_b200 import _abi
    fn = _abi.load().bt_debug_fused_layernorm_policy
    for rows in (tiles * 128, tiles * 128 - 127):
        assert fn(rows, hidden, SMS, 1) == all_rows
        assert fn(rows, hidden, SMS, 0) == padded


@pytest.mark.parametrize("tiles,hidden,all_rows,padded", [
    (12, 768, 0, 0), (13, 768, 1, 0),                    # 144 and 156 tiles of 64 columns
    (20, 768, 1, 0), (21, 768, 1, 0), (22, 768, 1, 1),   # three fifths of 21 are 12, of 22 are 13
    (24, 768, 1, 1), (25, 768, 0, 1), (32, 768, 1, 1),   # 144 and 150 tiles of 128 columns; the line on row tiles
    (9, 1024, 0, 0), (10, 1024, 1, 0), (16, 1024, 1, 0), (17, 1024, 1, 1), (19, 1024, 0, 1), (38, 1024, 1, 1),
    (18, 512, 0, 0), (19, 512, 1, 0), (31, 512, 1, 0), (32, 512, 1, 1), (37, 512, 0, 1),
    (39, 256, 0, 0), (40, 256, 1, 1),
    (64, 320, 0, 0), (64, 1280, 0, 0),                   # widths without the fused kernels
])
def test_layernorm_inside_the_gemm_saves_a_second_wave_of_narrow_tiles(policy, tiles, hidden, all_rows, padded):
    from bytetransformer_b200 import _abi
    fn = _abi.load().bt_debug_fused_layernorm_choice
    for rows in (tiles * 128, tiles * 128 - 127):
        assert fn(rows, hidden, SMS, 1) == all_rows
        assert fn(rows, hidden, SMS, 0) == padded


@pytest.mark.parametrize("tiles,N,K,pair", [
    (74, 768, 3072, 0), (75, 768, 3072, 1),              # two waves of 192-column tiles
    (148, 768, 768, 0), (149, 768, 768, 1),              # four, where K is short
    (74, 512, 2048, 0), (75, 512, 2048, 1), (75, 512, 512, 1),
    (37, 1024, 4096, 0), (38, 1024, 4096, 1),
    (148, 256, 1024, 0), (149, 256, 1024, 1),
    (74, 256, 2048, 0), (75, 256, 2048, 1), (148, 256, 4096, 1),  # one column tile and a long K
])
def test_layernorm_gemm_on_sm_pairs(policy, tiles, N, K, pair):
    for rows in (tiles * 128, tiles * 128 - 127):
        assert policy(6, rows, N, K, SMS) == pair
