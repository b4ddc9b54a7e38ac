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


@pytest.mark.parametrize("bits", [3, 4, 5, 6, 8])
@pytest.mark.parametrize("out_dtype", ["bfloat16", "float32", "float16"])
@pytest.mark.parametrize("n", [3, 131071, 131075])
def test_decoded_values(lib_built, n, out_dtype, bits):
    """Both sides of the size from which a thread decodes 16 values, outputs on and off the 32-byte boundary."""
    from mflux_b200 import _lib, ops

    g = torch.Generator(device="cuda").manual_seed(n + bits)
    w = (torch.randn(n, 64, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    codes, scales, biases = ops.quantize_affine(w, 64, bits)
    dt = getattr(torch, out_dtype)
    out = ops.dequantize_affine(codes, scales, biases, 64, bits, dt)
    few = slice(0, n, max(1, n // 97))
    ref = quant.dequantize_affine(codes[few].cpu().numpy(), scales[few].cpu().float().numpy(),
                                  biases[few].cpu().float().numpy(), 64, bits)
    assert torch.equal(out[few].cpu(), torch.from_numpy(ref).to(dt))
    step = 16 // out.element_size()
    odd = torch.full((n * 64 + 2 * step,), 7.0, device="cuda", dtype=dt)
    rc = _lib.load().mfx_dequantize_affine(codes.data_ptr(), scales.data_ptr(), biases.data_ptr(), _lib.BF16, n, 64, bits, 64,
                                           odd.data_ptr() + 16, ops._dt(odd), ops._stream())
    assert rc == 0 and torch.equal(odd[step:-step].view(n, 64), out)
    assert (odd[:step] == 7.0).all() and (odd[-step:] == 7.0).all()
