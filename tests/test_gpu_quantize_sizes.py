"""The quantizer on both sides of the size from which a thread takes 32 values of a 16-bit weight, with a ragged last
block, every width, constant and tie-rich groups: codes, scales and biases equal the oracle's."""
import pytest
import torch

from oracle import quant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [3, 4, 5, 6, 8])
@pytest.mark.parametrize("dtype", ["bfloat16", "float16", "float32"])
@pytest.mark.parametrize("n", [1, 65535, 65539])
def test_equal_to_oracle(lib_built, n, dtype, bits):
    from mflux_b200 import ops

    g = torch.Generator().manual_seed(n + bits)
    w = torch.randn(n, 64, generator=g) * 0.02
    if n > 1:
        w[100:4100] = torch.randint(-16, 17, (4000, 64), generator=g) / 2      # quotients on half-way points
        w[5000], w[5001] = 0.25, 0.0
        w[-1, 0] = 3.0
    w = w.to(getattr(torch, dtype))
    codes, scales, biases = ops.quantize_affine(w.cuda(), 64, bits)
    pc, ps, pb = quant.quantize_affine(w, 64, bits, dtype={"bfloat16": "bf16", "float16": "f16", "float32": "f32"}[dtype])
    assert (codes.cpu().numpy() == pc).all()
    assert (scales.cpu().float().numpy() == ps).all() and (biases.cpu().float().numpy() == pb).all()
