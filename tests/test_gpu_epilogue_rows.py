"""Rows of the quantized linear's output and residual on 16- but not on 32-byte boundaries (the 32-byte accesses of the
epilogue do not apply), and row widths that end inside a 32-column chunk: the same values as on aligned rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("epi", [None, "gelu", "gate_residual", "swiglu"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [48, 304, 512])
def test_misaligned_rows_give_the_same_values(lib_built, bits, epi, dtype, n):
    from mflux_b200 import ops

    m, k = 150, 128
    step = 16 // torch.empty(0, dtype=dtype).element_size()      # elements per 16 bytes
    g = torch.Generator(device="cpu").manual_seed(n + bits)
    wq, s, b = ops.quantize_affine((torch.randn(n, k, generator=g) * 0.1).to(torch.bfloat16).cuda(), 64, bits)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(n, generator=g).to(torch.bfloat16).cuda()
    res = torch.randn(m, n, generator=g).to(dtype).cuda()
    n_out = n // 2 if epi == "swiglu" else n
    width = -(-n_out // (2 * step)) * 2 * step

    def run(offset, pad):
        """Output (and residual) at column `offset` of rows `width + pad` elements apart."""
        out = torch.full((m, width + pad), 7.0, dtype=dtype, device="cuda")
        kw = {}
        if epi == "gate_residual":
            r = torch.zeros(m, width + pad, dtype=dtype, device="cuda")
            r[:, offset:offset + n] = res
            kw = {"gate": bias[None], "residual": r[:, offset:offset + n]}
        ops.qlinear(x, wq, s, b, bias, bits=bits, epilogue=epi, out=out[:, offset:offset + n_out], **kw)
        assert (out[:, :offset] == 7.0).all() and (out[:, offset + n_out:] == 7.0).all()
        return out[:, offset:offset + n_out]

    want = run(0, 0)
    assert torch.isfinite(want.float()).all()
    for offset, pad in ((step, 2 * step), (0, step), (step, step)):
        assert torch.equal(run(offset, pad), want)
    assert ops.poll_device_status() == 0


@pytest.mark.parametrize("two_launches", [False, True])
@pytest.mark.parametrize("epi", [None, "gelu", "gelu_approx", "silu", "gate_residual", "swiglu"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m", [17, 287, 2 * 256 + 33, 3 * 256 + 128 + 63])
def test_warps_whose_last_rows_are_missing(lib_built, monkeypatch, two_launches, epi, dtype, m):
    """A last row tile that ends inside a warp's 32 rows: some lanes of the warp write, the others only take part in the
    collective accumulator loads. The same rows as from a call whose tiles are full, on a column count with whole and
    broken 32-column chunks."""
    from mflux_b200 import ops

    n, k = 528, 192
    g = torch.Generator(device="cpu").manual_seed(m)
    wq, s, b = ops.quantize_affine((torch.randn(n, k, generator=g) * 0.1).to(torch.bfloat16).cuda(), 64, 4)
    full = -(-m // 256) * 256
    x = torch.randn(full, k, generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(n, generator=g).to(torch.bfloat16).cuda()
    res = torch.randn(full, n, generator=g).to(dtype).cuda()
    monkeypatch.setattr(ops, "_scratch_bytes", lambda *a: 2 * n * k if two_launches else 0)

    def run(rows):
        kw = {"gate": bias[None], "residual": res[:rows]} if epi == "gate_residual" else {}
        return ops.qlinear(x[:rows], wq, s, b, bias, bits=4, epilogue=epi, out_dtype=dtype, **kw)

    got, want = run(m), run(full)
    assert ops.poll_device_status() == 0
    assert got.shape[0] == m and torch.isfinite(got.float()).all()
    assert torch.equal(got, want[:m])
