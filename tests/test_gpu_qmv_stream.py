"""Few rows over weights of 24 M (two or four rows) and 48 or 36 M (eight) and more: every share of a tile's pieces among
warps (1, 2, 4, 8), one and several rounds of tiles, a last tile of eight rows, a last piece of one group, activations with
row strides, against float64 on the packed weights. Bound: float32 sums of up to 15360 terms and, for 4 bits, the offset of
128 that is taken out again (2^-24 of 128 Sum |x| per group against a result of about 5 |x| sqrt(64) codes: 2e-5 in the worst
case, a tenth of it on average)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weight(n, k, bits):
    from mflux_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(n + k)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    q = ops.quantize_affine(w, 64, bits)
    return q, ops.prepare_qlinear(*q, bits), ops.dequantize_affine(*q, 64, bits, torch.float32).double()


@pytest.mark.parametrize("n,k,bits", [(49160, 1024, 4), (81928, 640, 4), (18432, 3072, 4), (9224, 3072, 8), (16392, 3072, 8), (20480, 3840, 8),
                                      (3072, 15360, 4), (2184, 12352, 8), (8200, 3136, 3), (12288, 3072, 6)])
def test_against_float64(lib_built, n, k, bits):
    from mflux_b200 import ops

    q, prepared, w = _weight(n, k, bits)
    g = torch.Generator(device="cuda").manual_seed(1)
    bias = torch.randn(n, device="cuda", generator=g)
    most = 8 if n * k >= (48 if bits <= 4 else 36) << 20 else 2 if bits <= 4 else 4
    for rows, epilogue in ((1, None), (2, "silu"), (3, None), (4, None), (5, None), (8, None), (9, None)):
        x = torch.randn(rows, k + 64, device="cuda", generator=g).to(torch.bfloat16)[:, 32:32 + k]
        ref = x.double() @ w.t() + bias.double()
        if epilogue:
            ref = torch.nn.functional.silu(ref)
        y = ops.qlinear(x, *q, bias, bits=bits, prepared=prepared, epilogue=epilogue, out_dtype=torch.float32)
        again = ops.qlinear(x, *q, bias, bits=bits, prepared=prepared, epilogue=epilogue, out_dtype=torch.float32)
        assert torch.equal(y, again)
        stream = rows <= 2 or (rows <= most and k <= 4096)  # where the rows fit beside the rings
        assert ((y.double() - ref).norm() / ref.norm()).item() <= (2e-5 if stream else 4e-3)
        b16 = ops.qlinear(x, *q, bias, bits=bits, prepared=prepared, epilogue=epilogue)
        assert torch.equal(b16, y.to(torch.bfloat16))


@pytest.mark.parametrize("n,k,bits", [(18432, 3072, 4), (18432, 3072, 8)])
def test_values_that_are_not_finite(lib_built, n, k, bits):
    from mflux_b200 import ops

    q, prepared, _ = _weight(n, k, bits)
    w = ops.dequantize_affine(*q, 64, bits).float()
    x = torch.randn(8, k, device="cuda").to(torch.bfloat16)
    x[0, 5], x[1, 70], x[2, 9] = float("inf"), -float("inf"), float("nan")
    x[3, 100], x[3, 101] = float("inf"), -float("inf")
    x[4, 3] = 3e38                                          # finite result, sums of the factored form are not
    x[5, 64:128] = 1e37
    ref = (x.double() @ w.double().t()).float()
    y = ops.qlinear(x, *q, bits=bits, prepared=prepared, out_dtype=torch.float32)
    assert torch.equal(torch.isnan(y), torch.isnan(ref))
    assert torch.equal(torch.isinf(y), torch.isinf(ref)) and torch.equal(y[torch.isinf(y)], ref[torch.isinf(ref)])
    fine = torch.isfinite(ref)
    assert ((y[fine].double() - ref[fine].double()).norm() / ref[fine].double().norm()).item() <= 4e-3


@pytest.mark.parametrize("n,k,bits,rows", [(9216, 3072, 4, (1, 2)), (9216, 3072, 4, (3, 5, 16)), (9216, 3072, 8, (1, 3, 4)),
                                           (20480, 3840, 4, (1, 4, 8)), (3072, 256, 4, (1, 8, 9, 16))])
def test_a_row_does_not_depend_on_the_others(lib_built, n, k, bits, rows):
    """Within the sizes that one kernel takes (include/mfx.h): equal bits with any rows beside it."""
    from mflux_b200 import ops

    q, prepared, _ = _weight(n, k, bits)
    x = torch.randn(16, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).to(torch.bfloat16)
    first = [ops.qlinear(x[:m], *q, bits=bits, prepared=prepared, out_dtype=torch.float32)[0] for m in rows]
    assert all(torch.equal(first[0], y) for y in first[1:])
