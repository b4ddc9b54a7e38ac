"""Which of the two attention kernels a call takes, by the library's size rule (host code; 148 SMs, as on a B200, also
where no device is present)."""
import pytest

from mflux_b200 import _lib

# (samples, heads, tokens), measured on a B200 at the power limit, pair / ping-pong kernel, us
TWO_TILES = [(4, 24, 4096),     # 839 / 791: 10.4 waves
             (2, 24, 3600),     # 351 / 329: an odd number of query tiles
             (2, 24, 8192),     # 1580 / 1474
             (16, 24, 1536),    # 551 / 520
             (2, 30, 1613),     # 103 / 98
             (37, 4, 1024),     # 102 / 98: four whole waves of the shortest sequence
             (1, 24, 4608),     # 266 / 241
             (1, 24, 4096),     # 224 / 206: 2.6 waves
             (2, 12, 4352),     # 244 / 223
             (1, 6, 4608),      # 76 / 70: less than a wave
             (1, 24, 1024)]     # 21.5 / 21.0
ONE_TILE = [(1, 24, 1023), (1, 6, 2500), (1, 12, 1024), (64, 24, 512)]


@pytest.mark.parametrize("shape", TWO_TILES + ONE_TILE)
def test_two_query_tiles_where_that_kernel_was_the_faster_one(lib_built, shape):
    batch, heads, seq = shape
    want = 2 if shape in TWO_TILES else 1
    assert _lib.load().mfx_fmha_query_tiles(seq, seq, batch, heads) == want


@pytest.mark.parametrize("args", [(0, 64, 1, 1), (64, 0, 1, 1), (64, 64, 0, 1), (64, 64, 1, 0), (1 << 40, 64, 1, 1)])
def test_sizes_that_are_not_valid(lib_built, args):
    assert _lib.load().mfx_fmha_query_tiles(*args) == 0
