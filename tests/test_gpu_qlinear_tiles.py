"""The tile widths of the quantized matmul (256, 192 and 128 output columns) on ragged rows, columns and depth, with the
epilogues that change the column count or read other operands, against the float32 oracle. With 74 CTA pairs 300 x 9224,
300 x 9472 and 1613 x 1928 take 256 columns, 600 x 4600 takes 192, the others 128."""
import pytest
import torch

from oracle import quant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("mnk", [(300, 9224, 192), (300, 9472, 64), (17, 4744, 192), (257, 136, 320), (600, 4600, 192),
                                 (300, 4736, 128), (1613, 1928, 448)])
@pytest.mark.parametrize("epi", [None, "gate_residual", "swiglu", "lora"])
def test_tile_widths(lib_built, bits, mnk, epi):
    from mflux_b200 import ops

    m, n, k = mnk
    if epi == "swiglu":
        n -= n % 16
    g = torch.Generator(device="cpu").manual_seed(m + n + bits)
    w = (torch.randn(n, k, generator=g) * 0.05).to(torch.bfloat16)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    b = torch.randn(n, generator=g).to(torch.bfloat16)
    wq, s, bi = ops.quantize_affine(w.cuda(), 64, bits)
    ref = torch.from_numpy(quant.qlinear(x, wq.cpu().numpy(), s.float().cpu().numpy(), bi.float().cpu().numpy(), b, 64,
                                         bits))
    kw = {}
    if epi == "gate_residual":
        gate, res = torch.randn(1, n, generator=g), torch.randn(m, n, generator=g)
        kw = {"epilogue": epi, "gate": gate.cuda(), "residual": res.cuda()}
        ref = res + gate * ref
    elif epi == "swiglu":
        kw = {"epilogue": epi}
        ref = torch.nn.functional.silu(ref[:, 0::2]) * ref[:, 1::2]
    elif epi == "lora":
        t = torch.zeros(m, 128, dtype=torch.bfloat16)
        lb = torch.zeros(n, 128, dtype=torch.bfloat16)
        t[:, :72] = torch.randn(m, 72, generator=g)
        lb[:, :72] = torch.randn(n, 72, generator=g) * 0.05
        kw = {"lora_t": t.cuda(), "lora_b": lb.cuda(), "lora_r": 72}
        ref = ref + t.float() @ lb.float().t()
    n_out = ref.shape[1]
    buf = torch.full((m + 3, n_out + 8), 7.0, dtype=torch.float32, device="cuda")
    y = ops.qlinear(x.cuda(), wq, s, bi, b.cuda(), bits=bits, out=buf[:m, :n_out], **kw)
    torch.cuda.synchronize()
    assert ops.poll_device_status() == 0
    assert (buf[m:] == 7.0).all() and (buf[:, n_out:] == 7.0).all()
    assert quant.rel_l2(y, ref.numpy()) <= 1e-2
