"""Codes of values at and a few ulps beside the half-way points between two codes, where a rounded product with the
reciprocal of the scale and the rounded quotient may differ, over scales from the subnormals to near overflow (where
the reciprocal is no normal number): bit for bit the oracle's."""
import numpy as np
import pytest
import torch

from oracle import quant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["mlx", "doc"])
@pytest.mark.parametrize("bits", [3, 4, 5, 6, 8])
@pytest.mark.parametrize("exponent", [-140, -126, -100, -60, -7, 0, 30, 90, 110])
def test_near_ties_match_the_oracle(lib_built, mode, bits, exponent):
    from mflux_b200 import ops

    rng = np.random.default_rng(bits * 1000 + exponent + 500)
    n, groups, bins = 64, 4, 2 ** bits - 1
    unit = rng.uniform(1.0, 2.0, (n, groups, 1)) * 2.0 ** exponent
    half = rng.integers(0, bins, (n, groups, 64)) + 0.5
    half[..., 0], half[..., 1] = 0.0, bins                       # the group's edges span exactly `bins` units
    w = ((half - rng.integers(0, bins + 1, (n, groups, 1))) * unit).astype(np.float32)
    nudge = rng.integers(-3, 4, w.shape)
    nudge[..., :2] = 0
    for _ in range(3):
        w = np.where(nudge > 0, np.nextafter(w, np.float32(np.inf)), np.where(nudge < 0, np.nextafter(w, np.float32(-np.inf)), w))
        nudge = nudge - np.sign(nudge)
    w = w.reshape(n, groups * 64).astype(np.float32)
    pq, ps, pb = quant.quantize_affine(torch.from_numpy(w), 64, bits, mode=mode)
    wq, s, b = ops.quantize_affine(torch.from_numpy(w).cuda(), 64, bits, mode=mode)
    np.testing.assert_array_equal(s.cpu().numpy(), ps)
    np.testing.assert_array_equal(b.cpu().numpy(), pb)
    np.testing.assert_array_equal(wq.cpu().numpy(), pq)
