"""Attention calls on both sides of the choice between the two kernels (half a wave, one wave, a part-filled second and
third wave, an odd number of 128-query tiles, the shortest key lengths of either), with and without a key-padding bias,
against float64; which kernel a size takes is asserted first. The bound is the bf16 rounding of P and of the output (2^-9 each, relative) over averages of values:
5e-3 in the 2-norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("batch,heads,seq,tiles", [(1, 18, 1024, 1), (1, 20, 1024, 2), (1, 20, 1023, 1), (1, 30, 2047, 1),
                                                   (1, 30, 2048, 2), (1, 12, 2400, 1), (2, 6, 2500, 2), (1, 24, 4096, 2),
                                                   (18, 4, 1024, 2), (2, 24, 1536, 2)])
def test_both_sides_of_the_choice(lib_built, monkeypatch, bias, batch, heads, seq, tiles):
    from mflux_b200 import _lib, ops

    monkeypatch.delenv("MFX_FMHA_KERNEL", raising=False)
    assert _lib.load().mfx_fmha_query_tiles(seq, seq, batch, heads) == tiles
    g = torch.Generator(device="cuda").manual_seed(heads * seq)
    qkv = torch.randn(batch, seq, 3 * heads * 128, device="cuda", generator=g).to(torch.bfloat16)
    kb = None
    if bias:
        kb = torch.zeros(batch, seq, device="cuda")
        kb[:, seq - seq // 5:] = -1e9
    out = ops.fmha(qkv, heads, key_bias=kb)
    assert ops.poll_device_status() == 0
    for b, h in {(0, 0), (batch - 1, heads - 1)}:
        q, k, v = (qkv[b, :, (i * heads + h) * 128:(i * heads + h + 1) * 128].double() for i in range(3))
        s = q @ k.t() * 128 ** -0.5
        if bias:
            s = s + kb[b].double()
        ref = torch.softmax(s, dim=-1) @ v
        got = out[b, :, h * 128:(h + 1) * 128].double()
        assert ((got - ref).norm() / ref.norm()).item() <= 5e-3
