"""Epilogue activations against float64 on the whole range a layer output can take.

The quantized matmul is made an identity on its first 64 columns of x (codes of one 1 per row), so that the layer's
float32 output is f(x[:, n] + bias[n]) with an exactly known argument.
"""
import numpy as np
import pytest
import torch
from scipy import special

pytestmark = pytest.mark.gpu

N = 64


def _layer(x, epilogue, bias=None, two_launches=False):
    """f(x) in float32 and x as the layer sees it, both as float64 arrays."""
    from mflux_b200 import ops

    w = torch.eye(N, N)          # one group per row: min 0, max 1, so code 15 * (1 / 15) + 0 is 1 up to one rounding
    wq, s, b = ops.quantize_affine(w.cuda(), 64, 4)
    x = x.reshape(-1, N).to(torch.bfloat16).cuda()
    bias = None if bias is None else bias.cuda()
    with pytest.MonkeyPatch.context() as m:
        m.setattr(ops, "_scratch_bytes", lambda *a: 2 * N * N if two_launches else 0)
        y, plain = (ops.qlinear(x, wq, s, b, bias, bits=4, epilogue=e, out_dtype=torch.float32)
                    for e in (epilogue, None))
    assert ops.poll_device_status() == 0
    return y.cpu().double().numpy(), plain.cpu().double().numpy()


def _exact(name, v):
    if name == "gelu":
        return 0.5 * v * special.erfc(-v / np.sqrt(2.0))
    if name == "gelu_approx":
        return v * special.expit(2.0 * np.sqrt(2.0 / np.pi) * (v + 0.044715 * v ** 3))
    return v * special.expit(v)


@pytest.mark.parametrize("two_launches", [False, True])
@pytest.mark.parametrize("name", ["gelu", "gelu_approx", "silu"])
def test_activation_over_the_whole_range(lib_built, name, two_launches):
    """The largest error. GELU forms, v / 2 (1 + g): g's argument is off by at most five roundings, which erf and tanh
    pass on at most 0.49 times, g itself by 2 units in the last place, the sum by one rounding and the two products by
    one each: 3.2 x 2^-23 |v| with roundings of 2^-24. SiLU: exp is off by 2 + 1.16 |v| units, e^-|v| of which reach the
    result, and two roundings more: 2.5 x 2^-23 |v|. 2^-21 |v| holds for all, whatever v."""
    x = torch.cat([torch.linspace(-12, 12, 64 * 255), torch.linspace(-0.5, 0.5, 64 * 64),
                   torch.tensor([0.0, -0.0, 100.0, -100.0, 1e4, -1e4, 3e38, -3e38]).repeat(8)])
    y, v = _layer(x, name, two_launches=two_launches)
    assert np.isfinite(y).all() and np.abs(v).max() > 2e38
    err = np.abs(y - _exact(name, v))
    assert (err <= 2.0 ** -21 * np.abs(v)).all(), (err / np.maximum(np.abs(v), 1e-30)).max()


@pytest.mark.parametrize("two_launches", [False, True])
@pytest.mark.parametrize("name", ["gelu", "gelu_approx", "silu"])
def test_small_arguments_keep_float32_accuracy(lib_built, name, two_launches):
    """The usual error where layer outputs mostly lie. A chain of n float32 roundings, each of root mean square 2.5e-8
    (half a unit in the last place, evenly spread, over all mantissas), is off by sqrt(n) times that in the 2-norm; six
    cover each of the three formulas."""
    x = torch.randn(64 * 512, generator=torch.Generator().manual_seed(7)) * 0.3
    y, v = _layer(x, name, two_launches=two_launches)
    ref = _exact(name, v)
    assert np.linalg.norm(y - ref) / np.linalg.norm(ref) <= 2.5e-8 * np.sqrt(6)


@pytest.mark.parametrize("two_launches", [False, True])
@pytest.mark.parametrize("name", ["gelu", "gelu_approx", "silu"])
def test_infinities_and_nan(lib_built, name, two_launches):
    """Each formula written out in float32: +inf stays, -inf is inf * 0 or inf / inf, NaN stays."""
    bias = torch.zeros(N)
    bias[:3] = torch.tensor([float("inf"), -float("inf"), float("nan")])
    y, _ = _layer(torch.randn(64 * 40, generator=torch.Generator().manual_seed(8)), name, bias, two_launches)
    assert (y[:, 0] == np.inf).all() and np.isnan(y[:, 1:3]).all() and np.isfinite(y[:, 3:]).all()
