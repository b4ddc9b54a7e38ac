"""The tile widths of the quantized matmul (256, 192 and 128 output columns) on ragged rows, columns and depth, with the
epilogues that change the column count or read other operands: small grids against the float32 oracle, and grids that
give a CTA pair three tiles and more, where accumulators, rings and bias vectors are used in turn, bit for bit against
the two-launch form. Which width a size takes is asserted, so that a changed rule cannot leave a width untested."""
import pytest
import torch

from oracle import quant

pytestmark = pytest.mark.gpu

PAIRS = 74      # CTA pairs of a B200


def _width_and_tiles(rows, batch, n, bits):
    """Output columns of a tile in the one-launch form, and how many tiles the call has."""
    from mflux_b200 import _lib

    width = _lib.load().mfx_qlinear_tile_columns(rows, batch, n, bits)
    return width, batch * -(-rows // 256) * -(-n // width)


def _operands(m, n, k, bits, lora=0, batch=1):
    from mflux_b200 import ops

    g = torch.Generator(device="cpu").manual_seed(m + n + bits)
    w = (torch.randn(n, k, generator=g) * 0.05).to(torch.bfloat16)
    x = torch.randn(batch, m, k, generator=g).to(torch.bfloat16)
    b = torch.randn(n, generator=g).to(torch.bfloat16)
    wq, s, bi = ops.quantize_affine(w.cuda(), 64, bits)
    t = torch.zeros(batch, m, 128, dtype=torch.bfloat16)
    lb = torch.zeros(n, 128, dtype=torch.bfloat16)
    t[..., :lora] = torch.randn(batch, m, lora, generator=g)
    lb[:, :lora] = torch.randn(n, lora, generator=g) * 0.05
    return g, x, b, (wq, s, bi), t, lb


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("mnk,width", [((300, 9224, 192), 256), ((300, 9472, 64), 256), ((17, 4744, 192), 128),
                                       ((257, 136, 320), 128), ((600, 4600, 192), 192), ((300, 4736, 128), 128),
                                       ((1613, 1936, 448), 256)])
@pytest.mark.parametrize("epi", [None, "gate_residual", "swiglu", "lora"])
def test_tile_widths(lib_built, bits, mnk, width, epi):
    from mflux_b200 import ops

    m, n, k = mnk
    if epi == "swiglu":
        n -= n % 16
    assert _width_and_tiles(m, 1, n, bits)[0] == width
    g, x, b, (wq, s, bi), t, lb = _operands(m, n, k, bits, 72)
    x, t = x[0], t[0]
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
        kw = {"lora_t": t.cuda(), "lora_b": lb.cuda(), "lora_r": 72}
        ref = ref + t.float() @ lb.float().t()
    n_out = ref.shape[1]
    buf = torch.full((m + 3, n_out + 8), 7.0, dtype=torch.float32, device="cuda")
    y = ops.qlinear(x.cuda(), wq, s, bi, b.cuda(), bits=bits, out=buf[:m, :n_out], **kw)
    torch.cuda.synchronize()
    assert ops.poll_device_status() == 0
    assert (buf[m:] == 7.0).all() and (buf[:, n_out:] == 7.0).all()
    assert quant.rel_l2(y, ref.numpy()) <= 1e-2


# (rows, samples, columns, width): one sample and several, whole and ragged last tiles in both directions
WAVES = [(99 * 256 - 100, 1, 512, 256), (50 * 256 - 3, 2, 456, 256), (99 * 256 - 31, 1, 384, 192),
         (33 * 256 - 7, 3, 360, 192), (200 * 256 - 65, 1, 128, 128), (40 * 256 - 129, 5, 112, 128)]


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("rows,batch,n,width", WAVES)
@pytest.mark.parametrize("k", [64, 320])
@pytest.mark.parametrize("epi", [None, "gelu_approx", "gate_residual", "lora"])
def test_three_tiles_per_pair_match_the_two_launch_form(lib_built, monkeypatch, bits, rows, batch, n, width, k, epi):
    """One and three 128-k stages per tile: odd counts, so that rings and teams start every tile elsewhere. All rows,
    to the bit: same bf16 weights, same order of products, same epilogue."""
    from mflux_b200 import ops

    got_width, tiles = _width_and_tiles(rows, batch, n, bits)
    assert got_width == width and tiles > 2 * PAIRS
    g, x, b, (wq, s, bi), t, lb = _operands(rows, n, k, bits, 72 if epi == "lora" else 0, batch)
    kw = {"out_dtype": torch.float32}
    if epi == "gate_residual":
        kw = {"epilogue": epi, "gate": torch.randn(batch, n, generator=g).cuda(),
              "residual": torch.randn(batch, rows, n, generator=g).cuda()}
    elif epi == "lora":
        kw |= {"lora_t": t.cuda(), "lora_b": lb.cuda(), "lora_r": 72}
    elif epi:
        kw |= {"epilogue": epi}
    x, b, outs = x.cuda(), b.cuda(), []
    for need in (0, 2 * n * k):
        monkeypatch.setattr(ops, "_scratch_bytes", lambda *a, need=need: need)
        outs.append(ops.qlinear(x, wq, s, bi, b, bits=bits, **kw))
    assert ops.poll_device_status() == 0
    assert torch.isfinite(outs[0]).all() and torch.equal(*outs)
    if epi is None:
        wd = ops.dequantize_affine(wq, s, bi, 64, bits, torch.float32).cpu()
        ref = x[:, ::97].float().cpu() @ wd.t() + b.float().cpu()
        assert quant.rel_l2(outs[0][:, ::97], ref.numpy()) <= 1e-2
