"""Epilogue activations against float64 on the whole range a layer output can take.

The quantized matmul is made an identity on its first 64 columns of x (codes of one 1 per row), so that the layer's
float32 output is f(x[:, n] + bias[n]) with an exactly known argument.
"""
import numpy as np
import pytest
import torch
from scipy import special

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["gelu", "gelu_approx", "silu"])
def test_activation_over_the_whole_range(lib_built, name):
    from mflux_b200 import ops

    n = k = 64
    w = torch.eye(n, k)          # one group per row: min 0, max 1, so code 15 * (1 / 15) + 0 is exactly 1
    wq, s, b = ops.quantize_affine(w.cuda(), 64, 4)
    wd = ops.dequantize_affine(wq, s.to(torch.bfloat16).float(), b.to(torch.bfloat16).float(), 64, 4, torch.float32)
    x = torch.cat([torch.linspace(-12, 12, 64 * 255), torch.linspace(-0.5, 0.5, 64 * 64),
                   torch.tensor([0.0, -0.0, 100.0, -100.0, 1e4, -1e4, 3e38, -3e38]).repeat(8)])
    x = x.reshape(-1, k).to(torch.bfloat16)
    y = ops.qlinear(x.cuda(), wq, s, b, None, bits=4, epilogue=name, out_dtype=torch.float32).cpu().double().numpy()
    assert ops.poll_device_status() == 0
    plain = ops.qlinear(x.cuda(), wq, s, b, None, bits=4, out_dtype=torch.float32).cpu().double().numpy()
    assert np.isfinite(y).all() and float(wd.abs().max()) > 0.9
    if name == "gelu":
        ref = 0.5 * plain * special.erfc(-plain / np.sqrt(2.0))
    elif name == "gelu_approx":
        u = np.sqrt(2.0 / np.pi) * (plain + 0.044715 * plain ** 3)
        ref = plain * special.expit(2.0 * u)
    else:
        ref = plain * special.expit(plain)
    # float32 evaluation: the polynomial's 3e-7 plus a few roundings, and an exponent whose rounding grows with its
    # size (2^-24 of up to 126): 1e-5 relative; below 1e-30 the flushed tail counts as zero
    err = np.abs(y - ref) / np.maximum(np.abs(ref), 1e-30)
    assert err.max() <= 1e-5, (err.max(), plain.flat[err.argmax()])
