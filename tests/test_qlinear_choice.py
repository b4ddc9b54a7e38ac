"""Which form of the quantized linear a call takes, by the size rules of the library (host code; 74 CTA pairs, as on a
B200, also where no device is present)."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

from mflux_b200 import _lib

ROOT = Path(__file__).resolve().parent.parent


# (rows, samples, N, K, bits), measured on a B200, one launch / two launches, us
TWO_LAUNCHES = [(2816, 1, 9216, 3072, 8),      # 153 / 145
                (4096, 1, 3840, 10240, 8),     # 324 / 300
                (4213, 2, 20480, 3840, 8),     # 1170 / 1034
                (18432, 1, 3072, 3072, 4),     # 282 / 269
                (4608, 16, 12288, 3072, 4)]    # 36864 rows 2154 / 2082
ONE_LAUNCH = [(2560, 1, 3840, 10240, 8),       # 179 / 233: 150 wide tiles, 2.03 waves
              (2600, 1, 3840, 3840, 8),        # 75.7 / 81.6
              (3328, 1, 3072, 12288, 8),       # 243 / 255
              (3200, 1, 3072, 3072, 4),        # 49.1 / 66.4
              (3072, 1, 6144, 4096, 4),        # 123 / 132
              (4608, 1, 3072, 3072, 4),        # 71.2 / 75.5
              (36864, 1, 3840, 10240, 4),      # 2233 / 2444: the bf16 weight needs a second pass
              (1024, 1, 12288, 3072, 8)]


@pytest.mark.parametrize("shape", TWO_LAUNCHES + ONE_LAUNCH)
def test_two_launches_where_they_were_the_faster_form(lib_built, shape):
    rows, batch, n, k, bits = shape
    want = 2 * n * k if shape in TWO_LAUNCHES else 0
    assert _lib.load().mfx_qlinear_scratch_bytes_batch(rows, batch, n, k, bits) == want


def test_rows_of_short_samples_are_counted_in_their_own_tiles(lib_built):
    """64 samples of 60 rows fill 64 row tiles, 3840 rows of one sample 15."""
    lib = _lib.load()
    n, k = 9216, 3072
    for rows, batch, tiles in ((60, 64, 64), (3840, 1, 15), (257, 8, 16)):
        for bits in (4, 8):
            assert (lib.mfx_qlinear_scratch_bytes_batch(rows, batch, n, k, bits)
                    == lib.mfx_qlinear_scratch_bytes(256 * tiles, n, k, bits))


@pytest.mark.parametrize("args", [(0, 1, 64, 64, 4), (64, 0, 64, 64, 4), (64, 1, 0, 64, 4), (64, 1, 64, 100, 4),
                                  (64, 1, 64, 64, 7), (1 << 40, 1, 64, 64, 4), (1 << 30, 1 << 20, 1 << 30, 64, 8)])
def test_sizes_that_a_call_refuses_need_no_scratch(lib_built, args):
    assert _lib.load().mfx_qlinear_scratch_bytes_batch(*args) == 0


@pytest.mark.parametrize("rows,batch,n,bits,width", [
    (512, 1, 3072, 4, 128), (512, 1, 3072, 8, 128),        # few tiles: 61.9 / 55.0 / 41.6 us at 256 / 192 / 128 (K 12288)
    (1613, 1, 3840, 8, 192),                               # 128 / 113 / 118 us (K 10240)
    (1613, 1, 20480, 4, 256), (1613, 1, 20480, 8, 256),    # 191 / 210 / 227 and 218 / 226 / 234 us (K 3840)
    (16, 3, 64, 4, 128)])
def test_tile_width_by_waves(lib_built, rows, batch, n, bits, width):
    assert _lib.load().mfx_qlinear_tile_columns(rows, batch, n, bits) == width


@pytest.mark.parametrize("args", [(0, 1, 64, 4), (64, 0, 64, 4), (64, 1, 0, 4), (64, 1, 64, 7), (1 << 40, 1, 64, 4)])
def test_no_tile_width_for_sizes_that_a_call_refuses(lib_built, args):
    assert _lib.load().mfx_qlinear_tile_columns(*args) == 0


def test_no_scratch_where_the_tensor_memory_kernel_takes_the_calls(lib_built):
    """The scratch would be allocated for nothing and counted as a launch. MFX_QMM_KERNEL is read once per process."""
    code = ("from mflux_b200 import ops; "
            "print(ops._scratch_bytes(18432, 1, 3072, 3072, 4), ops._scratch_bytes(4608, 16, 9216, 3072, 8))")
    for kernel, want in (("tmem", "0 0"), ("", f"{2 * 3072 * 3072} {2 * 9216 * 3072}")):
        env = {**os.environ, "MFX_QMM_KERNEL": kernel}
        out = subprocess.run([sys.executable, "-c", code], env=env, cwd=ROOT, capture_output=True, text=True, check=True)
        assert out.stdout.strip() == want
